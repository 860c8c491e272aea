"""Solves of more than one cycle: what maxiter counts, and the results of
restarted solves."""
import numpy as np
import pytest

from oracle import simulation_fp64
from pyheartsim_b200 import _lib, instance, synthetic
from pyheartsim_b200.engine import BatchedEngine
from pyheartsim_b200.simulation import simulation_gpu
from tests import gpu_cases

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


def _steps(case, dtype, restart, steps, *, full=False, variant=None, tol=1e-6, atol=1e-12):
    """(u after ``steps`` steps, info) of one case in an engine of its own."""
    (n, P, geom, sp, ap), pdur = case
    inst = instance.compile_instance(n, P, geom, dict(sp), dict(ap), full_cycles=full, tol=tol, atol=atol, restart=restart,
                                     pacing_duration=pdur, max_steps=steps)
    with BatchedEngine(_lib.PREC_F32 if dtype == np.float32 else _lib.PREC_F64) as eng:
        if variant is not None:
            eng.configure(variant=variant)
        s = eng.add(inst)
        eng.advance(steps)
        u, _, _ = eng.state(s)
        return u.astype(np.float64), eng.info(s)


_CASES = {"sheet": lambda: gpu_cases.sheet_ms(), "shell": lambda: gpu_cases.small_shell_ms(),
          "fibres": lambda: gpu_cases.small_shell_ms_fibres()}


# Early exit in several cycles: the update into x, the check that takes b from the
# pairs, the next cycle from its residual.  Variants 5 and 6 (FP32) stage the update.
@pytest.mark.parametrize("name", list(_CASES))
@pytest.mark.parametrize("dtype,variant", [(np.float32, None), (np.float32, 0), (np.float32, 5), (np.float32, 6),
                                           (np.float64, None)])
@pytest.mark.parametrize("restart", [2, 3, 4])
def test_restarted_early_exit(name, dtype, variant, restart, cuda_device):
    case, steps, tol = _CASES[name](), 8, 1e-6
    u, info = _steps(case, dtype, restart, steps, variant=variant, tol=tol)
    uo, io = _steps(case, np.float64, 50, steps, full=True, tol=1e-13, atol=0.0)
    assert info["max_arnoldi"] > restart and info["nonconverged"] == 0 and info["status"] == 0
    assert io["nonconverged"] == 0
    # a step is off by at most tol ||b|| (|A^-1| near 1), ||b|| <= sqrt(excited voxels);
    # the upstroke amplifies an error by exp(0.05 / 0.3) a step at most (tau_in 0.3), the
    # sum of 8 steps is below 16; FP32 rounding is 6e-8 a step
    excited = np.count_nonzero(uo > 1e-3)
    assert 0 < excited and uo.max() <= 1.0
    eps = 6e-8 if dtype == np.float32 else 1e-16
    np.testing.assert_allclose(u, uo, rtol=0, atol=16 * (tol * np.sqrt(excited) + eps))


# One full-cycle step from rest, random voxels paced (r0 of the order of b, so the
# cycle that ends at rounding level is followed by a few columns more), and one
# whose cycles are too short to get there: the true residual of the result
@pytest.mark.parametrize("name", list(_CASES))
@pytest.mark.parametrize("restart", [50, 30, 8])
def test_full_cycles_true_residual(name, restart, cuda_device):
    (n, P, geom, sp, ap), _ = _CASES[name]()
    s1 = np.flatnonzero(np.random.default_rng(3).random(n) < 0.3)
    ap = dict(ap, s1_pacing_voxel_id=s1)
    u, info = _steps(((n, P, geom, sp, ap), 1.0), np.float64, restart, 1, full=True, tol=1e-13, atol=0.0)
    assert info["nonconverged"] == 0 and info["solves"] == 1
    J = np.zeros(n)
    J[s1] = 1.0
    us, _ = simulation_fp64.rk4(0, np.zeros(n), np.ones(n), P, J, sp["dt"])
    L = simulation_fp64.laplacian(P, geom["neighbor_id_2d"], geom["Delta"])
    b = us + sp["dt"] / 2 * (L @ us)
    r = b - (u - sp["dt"] / 2 * (L @ u))
    r0 = b - (us - sp["dt"] / 2 * (L @ us))
    assert np.linalg.norm(r0) > 0.1 * np.linalg.norm(b)
    # restart 8 stops at tol; the others at the rounding of the residual itself (a row adds up
    # to 20 terms of |A| |u|, below 4 |b|: 20 * 1.1e-16 * 4 would be the worst row, the norm over
    # random signs is sqrt(20) of it) and of u* on the two sides
    np.testing.assert_array_less(np.linalg.norm(r), (2e-15 if restart > 8 else 2e-13) * np.linalg.norm(b))


# Anisotropic rows, where the interval of the Chebyshev basis is a heuristic: the
# columns and the results of Arnoldi (restart 21, early exit, dt 0.2: beyond the rule)
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_chebyshev_and_arnoldi_agree_on_fibre_rows(dtype, cuda_device):
    steps = 20
    (n, P, geom, sp, ap), pdur = gpu_cases.small_shell_ms(dt=0.2, fibres=True)
    ub, ib = _steps(((n, P, geom, sp, ap), pdur), dtype, 21, steps, tol=1e-7, atol=1e-5)
    ua, ia = _steps(((n, P, geom, sp, ap), pdur), dtype, 20, steps, tol=1e-7, atol=1e-5)
    assert ia["nonconverged"] == ib["nonconverged"] == 0 and ia["max_arnoldi"] <= 20
    # the same spaces and the same test: the counts differ where an estimate falls on the tolerance
    assert abs(ia["arnoldi_steps"] - ib["arnoldi_steps"]) <= max(2, 0.02 * ib["arnoldi_steps"])
    # each solve leaves a residual of at most 1e-5 (atol) or 1e-7 ||b||, below 1e-5: twice that per step
    # and an upstroke's growth of exp(0.2 / 0.3) a step, in sum below 1.2e6 over 20 steps at worst; the
    # excited voxels here take under 5 steps to rise, 60 in sum
    np.testing.assert_allclose(ua, ub, rtol=0, atol=20 * 60 * 2e-5)
