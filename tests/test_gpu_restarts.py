"""Solves of more than one cycle: what maxiter counts, and the results of
restarted solves."""
import numpy as np
import pytest

from pyheartsim_b200 import _lib, instance, synthetic
from pyheartsim_b200.engine import BatchedEngine
from pyheartsim_b200.simulation import simulation_gpu

pytestmark = pytest.mark.gpu


def _plane_front(hg, steps):
    """A 64 x 64 sheet paced along one edge, its diffusion scaled so that the
    eigenvalues of dt/2 (-L) lie in [0, 2 hg] (1.25 at scale 1)."""
    ijk = synthetic.sheet(64, 64)
    s1 = np.where(ijk[:, 0] < 5)[0]
    return synthetic.make_case(ijk, 0.4, 0, 0.05, 1.0, s1, flag=4, c_scale=np.full(len(ijk), hg / 0.625))


# Column counts of Arnoldi GMRES(20) in these solves: at most 47, 20, 40 and 60;
# Chebyshev cycles lose their Gram matrix after 10-17 columns in all of them
@pytest.mark.parametrize("dtype,hg,tol,maxiter", [(np.float32, 60.0, 1e-5, 60), (np.float64, 3.0, 1e-9, 20),
                                                  (np.float64, 15.0, 1e-9, 40), (np.float64, 30.0, 1e-9, 60)])
def test_short_cycles_do_not_use_up_maxiter(dtype, hg, tol, maxiter, cuda_device):
    steps = 4
    n, P, geom, sp, ap = _plane_front(hg, steps)
    u, h, t, info = simulation_gpu.compute(n, P, geom, dict(sp), dict(ap), pacing_duration=1.0, dtype=dtype, fast=True,
                                           tol=tol, atol=1e-12, restart=20, maxiter=maxiter, max_steps=steps,
                                           return_info=True)
    assert info["nonconverged"] == 0 and info["solves"] == steps
    uo, ho, to = simulation_gpu.compute(n, P, geom, dict(sp), dict(ap), pacing_duration=1.0, max_steps=steps,
                                        tol=1e-13, atol=0.0)
    assert u.shape == uo.shape and u.shape[0] >= 1
    # |A^-1| <= 1: a step is off by at most tol ||b||, ||b|| < 2 sqrt(n); rounding of FP32
    # is 6e-8 of that
    np.testing.assert_allclose(u, uo, rtol=0, atol=steps * tol * 2 * 64 + (1e-5 if dtype == np.float32 else 0))


def _tiny_state(scale, full, tol):
    """A resting Mitchell-Schaeffer strip decayed to ``scale``, its time
    constants (and so its decay) different from voxel to voxel."""
    ijk = synthetic.sheet(40, 12)
    n, P, geom, sp, ap = synthetic.make_case(ijk, 0.4, 0, 0.05, 1.0, [0], flag=4)
    P = P.copy()
    P[:, 18] = np.where(ijk[:, 0] % 7 < 3, 0.02, 6.0)      # tau_out
    ap = dict(ap, s1_pacing_voxel_id=np.zeros(0, np.int64))
    inst = instance.compile_instance(n, P, geom, sp, ap, full_cycles=full, tol=tol, atol=0.0, restart=50 if full else 20,
                                     pacing_duration=0.0, max_steps=1, guess=0)
    inst.u0 = scale
    with BatchedEngine(_lib.PREC_F64) as eng:
        s = eng.add(inst)
        eng.advance(1)
        u, _, _ = eng.state(s)
        return u, eng.info(s)


# The equations are linear at rest to far below rounding (the cubic term is u^2 of
# the linear one), so the scaled result does not depend on the scale: at 2^-400 and
# 2^-498 (u^2 is still a normal number) it is that at 2^-100
@pytest.mark.parametrize("full,tol", [(False, 1e-7), (False, 1e-12), (True, 1e-5)])
@pytest.mark.parametrize("exponent", [-164, -170, -400, -498])
def test_tiny_states_are_solved_like_small_ones(exponent, full, tol, cuda_device):
    u0, i0 = _tiny_state(2.0 ** -100, full, tol)
    u1, i1 = _tiny_state(2.0 ** exponent, full, tol)
    assert i1["status"] == 0 and i1["nonconverged"] == 0 and i1["solves"] == 1
    a, b = u0 * 2.0 ** 100, u1 * 2.0 ** -exponent
    assert 0.0 < a.min() < 0.9 * a.max()                   # a field with something to solve
    # both residuals are at most tol ||b|| (full cycles: far below), |A^-1| <= 1; rounding 1e-14
    np.testing.assert_allclose(b, a, rtol=0, atol=max(1e-14, (0.0 if full else 2 * tol) * np.linalg.norm(a)))
