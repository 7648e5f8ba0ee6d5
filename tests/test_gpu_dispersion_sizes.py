"""The dispersion image at the sizes where its kernels' tiles and folds can go
wrong, on a B200, against the numpy restatement: odd and even sample counts
(with even counts the spectrum is folded about nt/4), the smallest, counts
around the tiles of 32 frequencies and 64 traces, roots beyond shared memory."""
import numpy as np
import pytest

from oracle import dispersion

pytestmark = pytest.mark.gpu

# amplitudes are at most 1, returned in FP32 (rounding 6e-8) from FP64 sums over
# ntr traces of phases up to w x / c ~ 1e4 (2^-52 each: 2e-12): 1e-6 leaves room
# for bins whose |S| is small against the noise's rounding
TOL = 1e-6


@pytest.mark.parametrize("nt,ntr,nv", [(2, 1, 1), (3, 2, 3), (4, 3, 2), (5, 1, 65), (6, 65, 64),
                                       (62, 63, 7), (64, 64, 9), (127, 129, 66), (128, 33, 5),
                                       (130, 7, 130), (1001, 31, 3), (4097, 5, 4), (4098, 3, 2)])
def test_image_matches_numpy(mfdm, nt, ntr, nv):
    rng = np.random.default_rng([nt, ntr])
    g = rng.standard_normal((nt, ntr)).astype(np.float32)
    x = np.sort(rng.uniform(-2000.0, 2000.0, ntr))
    c_min, dc = 1400.0, 7.0
    c_max = c_min + dc * (nv - 1)
    f, v, a = mfdm.dispersion_image(g, x, 500.0, c_min, c_max, dc)
    S = np.fft.rfft(g.astype(np.float64), axis=0)
    P = np.conj(S) / np.abs(S)
    w = 2.0 * np.pi * f
    ref = np.abs((P[:, None, :] * np.exp(-1j * w[:, None, None] * x[None, None, :] / v[None, :, None])).sum(2)) / ntr
    assert a.shape == (nt // 2 + 1, nv)
    assert np.allclose(v, dispersion.velocities(c_min, c_max, dc))
    assert np.max(np.abs(a - ref)) <= TOL


def test_silent_traces_stay_silent(mfdm):
    """A trace of zeros has no phase: it adds nothing (but counts in the mean)."""
    rng = np.random.default_rng(3)
    g = rng.standard_normal((96, 4)).astype(np.float32)
    g[:, 2] = 0.0
    x = np.arange(4.0) * 10.0
    _, _, a = mfdm.dispersion_image(g, x, 500.0, 1500.0, 1510.0, 5.0)
    _, _, b = mfdm.dispersion_image(g[:, [0, 1, 3]], x[[0, 1, 3]], 500.0, 1500.0, 1510.0, 5.0)
    assert np.max(np.abs(a - 0.75 * b)) <= TOL
