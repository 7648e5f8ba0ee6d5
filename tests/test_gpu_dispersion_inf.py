"""Infinite and NaN samples in a gather's dispersion image on a B200: where the DFT
multiplies an infinite sample by the zero sine of the root 1 the trace has no phase
there and adds nothing, as a NaN sample's trace nowhere does."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-6  # as tests/test_gpu_dispersion_sizes.py: FP64 sums returned in FP32, at most 1


def images(mfdm, nt, t, value):
    rng = np.random.default_rng([nt, t])
    g = rng.standard_normal((nt, 5)).astype(np.float32)
    x = np.arange(5.0) * 10.0
    g[:, 3] = 0.0
    silent = mfdm.dispersion_image(g, x, 500.0, 1500.0, 1510.0, 5.0)[2]
    g[:, 3] = rng.standard_normal(nt)
    g[t, 3] = value
    return mfdm.dispersion_image(g, x, 500.0, 1500.0, 1510.0, 5.0)[2], silent


@pytest.mark.parametrize("nt", [64, 65, 130, 4098])
@pytest.mark.parametrize("value", [np.inf, -np.inf])
def test_infinite_first_sample(mfdm, nt, value):
    a, silent = images(mfdm, nt, 0, value)
    assert np.max(np.abs(a - silent)) <= TOL


@pytest.mark.parametrize("nt", [64, 130])
def test_infinite_middle_sample(mfdm, nt):
    a, silent = images(mfdm, nt, nt // 2, np.inf)  # its root is 1 at even frequencies
    assert np.max(np.abs(a[::2] - silent[::2])) <= TOL


@pytest.mark.parametrize("nt,t", [(64, 0), (64, 32), (65, 7), (130, 99)])
def test_nan_sample(mfdm, nt, t):
    a, silent = images(mfdm, nt, t, np.nan)
    assert np.max(np.abs(a - silent)) <= TOL
