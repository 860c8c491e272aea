"""Electrode analysis where its kernels' pieces begin and end: time steps split
over the parts of a CTA, neighbourhoods around the size of a warp's shared
memory, histories around the rows a thread loads at once."""
import ctypes

import numpy as np
import pytest

from oracle import analysis as oracle_analysis
from pyheartsim_b200 import _lib, analysis

pytestmark = pytest.mark.gpu

CV_RTOL = 1e-9     # SVD plane fit vs numpy's LAPACK lstsq, FP64


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("T", [2, 3, 32, 33, 34, 65, 1000])
@pytest.mark.parametrize("ne", [1, 31, 33])
def test_lat_parts(T, ne, dtype, cuda_device):
    rng = np.random.default_rng(T * 100 + ne)
    egm = rng.integers(-3, 4, size=(T, ne)).astype(dtype)         # many ties, within and across parts
    egm[rng.integers(0, T), 0] = np.nan                           # a NaN in some part
    if ne > 2 and T > 40:
        egm[40:, 1] = np.nan
        egm[5, 2] = np.inf
    with np.errstate(invalid="ignore"):
        want = oracle_analysis.compute_electrode_lat(egm)
    np.testing.assert_array_equal(analysis.compute_electrode_lat(egm), want)


@pytest.mark.parametrize("n", [3, 4, 5, 511, 512, 513])
def test_cv_neighbourhood_sizes(n, cuda_device):
    """All points within the radius of one another: m = n for each of them (512:
    the most a warp holds; 513: the general form), and a flat set (rank 3)."""
    rng = np.random.default_rng(n)
    for flat in (False, True):
        xyz = rng.uniform(0, 4, size=(n, 3))
        if flat:
            xyz[:, 2] = 0.8
        lat = xyz @ np.array([1.5, -0.7, 0.4]) + rng.normal(0, 0.05, n)
        v, m, mean = analysis.conduction_velocity(xyz, lat)
        vo, mo, meano = oracle_analysis.conduction_velocity(xyz, lat)
        np.testing.assert_array_equal(np.isnan(m), np.isnan(mo))
        np.testing.assert_allclose(v, vo, rtol=CV_RTOL, atol=0)
        np.testing.assert_allclose(m, mo, rtol=CV_RTOL, atol=0)


@pytest.mark.parametrize("is64", [False, True])
@pytest.mark.parametrize("S", [1, 15, 16, 17, 40])
def test_activation_rows(S, is64, cuda_device):
    import torch
    rng = np.random.default_rng(S)
    n, ld, k = 300, 307, 3
    hist = rng.uniform(0, 1, size=(S, ld)).astype(np.float64 if is64 else np.float32)
    hist[rng.uniform(size=hist.shape) < 0.02] = np.nan            # NaN is below the threshold
    d = torch.as_tensor(hist, device=cuda_device)
    times = torch.full((n, k), -1, dtype=torch.int32, device=cuda_device)
    counts = torch.zeros(n, dtype=torch.int32, device=cuda_device)
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    _lib.check(_lib.lib().phs_activation_times(S, n, p(d), ld, int(is64), 0.5, k, p(times), p(counts), None),
               "phs_activation_times")
    torch.cuda.synchronize()
    above = hist[:, :n] >= 0.5
    cross = above & ~np.vstack([np.zeros((1, n), bool), above[:-1]])
    np.testing.assert_array_equal(counts.cpu().numpy(), cross.sum(axis=0))
    want = np.full((n, k), -1, np.int32)
    for v in range(n):
        at = np.flatnonzero(cross[:, v])[:k]
        want[v, :at.size] = at
    np.testing.assert_array_equal(times.cpu().numpy(), want)
