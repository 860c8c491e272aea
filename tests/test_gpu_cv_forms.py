"""Conduction velocity where its two forms meet: neighbourhoods on both sides of
what a warp holds in one call, and electrode counts on both sides of the
number up to which warps search."""
import numpy as np
import pytest

from oracle import analysis as oracle_analysis
from pyheartsim_b200 import analysis

pytestmark = pytest.mark.gpu

CV_RTOL = 1e-9     # SVD plane fit vs numpy's LAPACK lstsq, FP64


def _fit(xyz, lat, i):
    """The plane fit of electrode i over the electrodes within 8 mm."""
    near = ((xyz - xyz[i]) ** 2).sum(axis=1) <= 64.0
    if near.sum() < 4:
        return np.full(3, np.nan)
    A = np.column_stack([xyz[near], np.ones(near.sum())])
    g = np.linalg.lstsq(A, lat[near], rcond=None)[0][:3]
    return g / (g @ g)


@pytest.mark.parametrize("dense", [512, 513, 700])
def test_dense_and_sparse_neighbourhoods_in_one_call(dense, cuda_device):
    rng = np.random.default_rng(dense)
    xyz = np.vstack([rng.uniform(0, 4, size=(dense, 3)), rng.uniform(20, 60, size=(300, 3)),
                     rng.uniform(100, 103, size=(513, 3))])[rng.permutation(dense + 813)]
    lat = xyz @ np.array([1.5, -0.7, 0.4]) + rng.normal(0, 0.05, len(xyz))
    v, m, mean = analysis.conduction_velocity(xyz, lat)
    vo, mo, meano = oracle_analysis.conduction_velocity(xyz, lat)
    np.testing.assert_array_equal(np.isnan(m), np.isnan(mo))
    np.testing.assert_allclose(v, vo, rtol=CV_RTOL, atol=0)
    np.testing.assert_allclose(m, mo, rtol=CV_RTOL, atol=0)
    np.testing.assert_allclose(mean, meano, rtol=CV_RTOL)


@pytest.mark.parametrize("n", [1 << 17, (1 << 17) + 1])
def test_electrode_counts_around_the_search_limit(n, cuda_device):
    rng = np.random.default_rng(n)
    side = (n / 40 * (4 / 3 * np.pi * 512)) ** (1 / 3)
    xyz = rng.uniform(0, side, size=(n, 3))
    xyz[1000:1600] = rng.uniform(-50, -46, size=(600, 3))          # a spot of its own, above 512 neighbours
    lat = xyz @ np.array([1.5, -0.7, 0.4]) + rng.normal(0, 0.05, n)
    v, m, mean = analysis.conduction_velocity(xyz, lat)
    for i in [0, 1000, 1599, n - 1, *rng.integers(0, n, size=60)]:
        want = _fit(xyz, lat, i)
        np.testing.assert_array_equal(np.isnan(v[i]), np.isnan(want))
        if not np.isnan(want).any():
            np.testing.assert_allclose(v[i], want, rtol=CV_RTOL, atol=0)
            np.testing.assert_allclose(m[i], np.linalg.norm(want), rtol=CV_RTOL)
