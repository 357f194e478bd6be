"""The radius outside which a step of hmax needs no error estimate (parrelray_b200/csrc/phys_stepper.cuh:cruise_radius, the
function itself compiled for the host) over energies, masses, spins, tolerances and step lengths, and the maxima of the
embedded difference that it is built on: at r >= 4M and s = h E / r <= 1/8, 0.8 M s^5 in x and 1.4 (M/r) E s^5 in p."""
import ctypes as C

import numpy as np
import pytest

from host_device import library
from test_error_skip import A, B4, B5, ks, null_momentum, rhs

SOURCE = r"""
#include "phys_stepper.cuh"
extern "C" float radius(float hmax, float atol, float E, float M, int fp32)
{
    prr::FrameParams fp;
    std::memset(&fp, 0, sizeof fp);
    fp.hmax = hmax; fp.atol = atol;
    return prr::cruise_radius(fp, E, M, fp32 ? prr::cruise_noise<float>() : prr::cruise_noise<double>());
}
"""


@pytest.fixture(scope="module")
def radius():
    lib = library(SOURCE)
    lib.radius.restype = C.c_float
    f = C.c_float
    return lambda hmax, atol, E, M, fp32=0: lib.radius(f(hmax), f(atol), f(E), f(M), int(fp32))


def states(rng, n, r, M, E):
    """Null states of energy E at Kerr-Schild radius r, every spin and direction."""
    a = M * rng.uniform(-1.0, 1.0, n)
    ct, ph = rng.uniform(-1, 1, n), rng.uniform(0, 2 * np.pi, n)
    st, R = np.sqrt(1 - ct * ct), np.sqrt(r * r + a * a)
    x = np.stack((R * st * np.cos(ph), R * st * np.sin(ph), r * ct))
    d = rng.normal(size=(3, n))
    d /= np.sqrt((d * d).sum(0))
    p, pt = null_momentum(d, ks(*x, M, a))
    return np.concatenate((x, p * E / np.abs(pt))), pt * E / np.abs(pt), a


def embedded(s, pt, M, a, h):
    k = []
    for row in A:
        z = s
        for c, kk in zip(row, k):
            z = z + s.dtype.type(c) * kk
        k.append(h * rhs(z, pt, M, a))
    return np.abs(sum(s.dtype.type(c5 - c4) * kk for c5, c4, kk in zip(B5, B4, k) if c5 != c4))


def test_maxima_of_the_embedded_difference():
    rng = np.random.default_rng(21)
    n = 300_000
    M = np.exp(rng.uniform(np.log(0.05), np.log(5.0), n))
    E = np.exp(rng.uniform(np.log(0.02), np.log(50.0), n))
    r = 4.0 * M * np.exp(rng.uniform(0.0, 3.0, n) * (rng.random(n) < 0.7))
    s = 0.125 * np.exp(rng.uniform(-2.5, 0.0, n) * (rng.random(n) < 0.7))
    y, pt, a = states(rng, n, r, M, E)
    e = embedded(y, pt, M, a, s * r / E)
    noise = 1e-14
    assert (e[:3].max(0) <= 0.8 * M * s**5 + noise * r).all()
    assert (e[3:].max(0) <= 1.4 * M / r * E * s**5 + noise * E).all()


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_no_estimate_is_needed_outside_the_radius(radius, dtype):
    """err < 0.9^5 of the scale's lower bound atol, where 0.9 h err^(-1/5) leaves h at hmax."""
    rng = np.random.default_rng(22)
    used = 0
    for _ in range(150):
        E, M = np.exp(rng.uniform(np.log(0.02), np.log(50.0))), np.exp(rng.uniform(np.log(0.02), np.log(5.0)))
        hmax, atol = np.exp(rng.uniform(np.log(0.01), np.log(1.0))), 10.0 ** rng.uniform(-9, -4)
        lo = radius(hmax, atol, E, M, dtype is np.float32)
        if not np.isfinite(lo):
            continue
        used += 1
        n = 2000
        r = float(lo) * np.exp(rng.uniform(0.0, 3.0, n) * (np.arange(n) % 2))
        y, pt, a = states(rng, n, r, M, E)
        c = lambda v: np.asarray(v, dtype=dtype)  # noqa: E731
        e = embedded(c(y), c(pt), c(M), c(a), c(hmax)).max(0)
        assert np.isfinite(e).all() and e.max() < 0.9**5 * atol, (E, M, hmax, atol, e.max())
    assert used >= (100 if dtype is np.float64 else 15)


def test_the_rule_refuses_what_rounding_spoils(radius):
    assert radius(0.1, 1e-6, 1.0, 1.0) < 40.0
    assert np.isinf(radius(0.1, 0.0, 1.0, 1.0)) and np.isinf(radius(0.1, 1e-9, 1.0, 1.0, 1)) and np.isinf(radius(0.1, 1e-6, np.nan, 1.0))
