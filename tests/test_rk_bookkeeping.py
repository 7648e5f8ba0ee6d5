"""The once-a-step RK4 bookkeeping (mfdm_device.cuh, rk_acc / rk_last / rk_once), restated in numpy float32.

A step accumulates once, in the second stage: acc = 2/3 U + (Y2 - U)/3 + w k2, and
U' = acc + Y4/3 + c k4, w and c close to dt/3 and dt/6 (rk_once). The weights come from the header, so they are checked as compiled.
"""
import os
import re

import numpy as np
import pytest

HEADER = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                      "marineseis-fdm-2d_b200", "csrc", "mfdm_device.cuh")
F = np.float32


def weight(name):
    num, den = re.search(rf"constexpr float {name} = ([0-9.]+)f / ([0-9.]+)f;", open(HEADER).read()).groups()
    return F(num) / F(den)


W, W2 = weight("kThird"), weight("kTwoThirds")


def fma(a, b, c):
    return F(np.float64(a) * np.float64(b) + np.float64(c))


def rk_acc(k, y, u, w):
    return fma(W2, u, fma(w, k, W * (y - u)))


def rk_last(k, y, acc, c):
    p = W * y
    s = acc + p
    return s + fma(c, k, (p - (s - acc)) + fma(W, y, -p))


def test_the_weights_of_the_old_state_sum_to_one():
    assert float(W) + float(W2) == 1.0
    assert abs(float(W) - 1.0 / 3.0) <= 2.0 ** -24


@pytest.mark.parametrize("seed", [0, 1, 2])
def test_a_constant_state_stays_constant(seed):
    """k = 0: U' may differ from U by the roundings of acc and of U' only, without drift."""
    u0 = np.random.default_rng(seed).standard_normal(4096).astype(F)
    u = u0.copy()
    for _ in range(100):
        u = rk_last(F(0), u, rk_acc(F(0), u, u, F(1e-4)), F(1e-4))
    # acc rounds to half an ulp of 2/3 U; adding Y4/3 exactly and rounding returns U itself
    # unless that half ulp reaches half an ulp of U: at most one ulp a step either way, and
    # it must not accumulate in one direction over the sample
    assert np.all(np.abs(u - u0) <= 100 * np.spacing(np.abs(u0)))
    assert abs(float(np.mean((u - u0) / np.spacing(np.abs(u0))))) <= 0.1


@pytest.mark.parametrize("z", [-0.5, -1e-3, 0.3])
def test_the_step_is_classical_rk4(z):
    """y' = lambda y with dt lambda = z: one step multiplies by the RK4 polynomial. Roundings: the
    stage inputs (weights 1/3, 1/3), acc, the result, and the weights' 2^-24: under 4 x 2^-24."""
    dt, lam = F(1e-3), F(z) / F(1e-3)
    zz = float(dt) * float(lam)
    u = np.random.default_rng(5).uniform(1.0, 2.0, 4096).astype(F)
    k1 = lam * u
    y2 = fma(dt / F(2), k1, u)
    k2 = lam * y2
    y3 = fma(dt / F(2), k2, u)
    c = F(0.5 * float(W) * float(dt))
    w = F(float(dt) - 1.5 * float(W) * float(dt) - float(c))
    acc = rk_acc(k2, y2, u, w)
    y4 = fma(dt, lam * y3, u)
    got = rk_last(lam * y4, y4, acc, c).astype(np.float64)
    want = u.astype(np.float64) * (1 + zz + zz ** 2 / 2 + zz ** 3 / 6 + zz ** 4 / 24)
    assert np.max(np.abs(got / want - 1)) <= 4 * 2.0 ** -24 * (1 + 4 * abs(zz))
