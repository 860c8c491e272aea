"""The step kernel's solver where its tiles, groups of tiles and choice of basis
change: instances around the tile length and beyond one tile per group, and the
Chebyshev-basis form against the Arnoldi one."""
import numpy as np
import pytest

from oracle import simulation_fp64
from pyheartsim_b200 import synthetic
from pyheartsim_b200.simulation import simulation_gpu
from tests import gpu_cases

pytestmark = pytest.mark.gpu


def _strip(n, steps, dt=0.05):
    ijk = synthetic.sheet(n, 1)
    s1 = np.where(ijk[:, 0] < 5)[0]
    return synthetic.make_case(ijk, 0.4, 0, dt, steps * dt, s1, flag=4)


def _compute(case, pdur, **kw):
    n, P, geom, sp, ap = case
    return simulation_gpu.compute(n, P, geom, dict(sp), dict(ap), pacing_duration=pdur, **kw)


# tiles hold 256 voxels in FP64
@pytest.mark.parametrize("n", [1, 2, 255, 256, 257, 1023, 1025])
def test_strips_around_the_tile_length(n, cuda_device):
    case = _strip(n, 60)
    u, h, t, lat = _compute(case, 2.0, return_lat=True)
    uo, ho, to, lato = simulation_fp64.compute(*case[:3], dict(case[3]), dict(case[4]), pacing_duration=2.0,
                                               record_lat=True)
    # rounding only (both solve to rounding level)
    np.testing.assert_allclose(u, uo, rtol=0, atol=1e-9)
    np.testing.assert_allclose(h, ho, rtol=0, atol=1e-9)
    np.testing.assert_array_equal(lat, lato)


# more tiles than groups: 444 groups of 256-voxel tiles (FP64), 640 of 512-voxel
# tiles (FP32; checked against the FP64 run, whose tiles are in groups of three)
def test_several_tiles_per_group(cuda_device):
    case, pdur = gpu_cases.sheet_ms(nx=340, ny=340, t_phys=1.5)
    u, h, t = _compute(case, pdur)
    uo, ho, to = simulation_fp64.compute(*case[:3], dict(case[3]), dict(case[4]), pacing_duration=pdur)
    assert u.shape[0] == 2          # steps 0 and 20
    np.testing.assert_allclose(u, uo, rtol=0, atol=1e-9)
    np.testing.assert_allclose(h, ho, rtol=0, atol=1e-9)
    case, pdur = gpu_cases.sheet_ms(nx=600, ny=600, t_phys=1.5)
    u, h, t = _compute(case, pdur)
    u32, h32, _ = _compute(case, pdur, dtype=np.float32, fast=True, tol=1e-7)
    # a residual of at most 1e-5 (atol) a step, over 21 steps; FP32 rounding is far below
    np.testing.assert_allclose(u32, u, rtol=0, atol=21e-5)
    np.testing.assert_allclose(h32, h, rtol=0, atol=21e-5)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_chebyshev_and_arnoldi_forms_agree(dtype, cuda_device):
    """dt 0.2: restart 20 uses the Chebyshev basis, restart 21 Arnoldi."""
    case, pdur = gpu_cases.sheet_ms(t_phys=8.0, dt=0.2)
    runs = [_compute(case, pdur, dtype=dtype, fast=True, tol=1e-7, restart=m, return_info=True, return_lat=True)
            for m in (20, 21)]
    (ua, ha, _, la, ia), (ub, hb, _, lb, ib) = runs
    assert ia["max_arnoldi"] <= 20 and ia["nonconverged"] == ib["nonconverged"] == 0
    # the same Krylov spaces and the same test: the column counts differ only where
    # an estimate falls on the tolerance itself
    assert abs(ia["arnoldi_steps"] - ib["arnoldi_steps"]) <= 0.02 * ib["arnoldi_steps"]
    # each solve leaves a residual of at most 1e-5 (atol): 40 steps of twice that
    np.testing.assert_allclose(ua, ub, rtol=0, atol=40 * 2e-5)
    np.testing.assert_allclose(ha, hb, rtol=0, atol=40 * 2e-5)
    assert np.abs(la.astype(np.int64) - lb).max() <= 1
