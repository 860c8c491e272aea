"""Solves of more than one cycle: what maxiter counts, and the results of
restarted solves."""
import numpy as np
import pytest

from pyheartsim_b200 import synthetic
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
