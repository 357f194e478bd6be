"""parrelray_b200/csrc/sphere_path.cuh, compiled for the host: no hit within the length it gives, where the points of a
ray are rounded to FP32 (small spheres far from the origin) and where a sphere reaches as far as the hole."""
import ctypes as C

import numpy as np
import pytest

from host_device import library
from test_error_skip import attempt, ks, null_momentum, rhs
from test_quick_steps import hit_distance, unit

F = np.float32

SOURCE = r"""
#include "sphere_path.cuh"
template <class T> static void each(int n, const double *c, double R, const T *p, const T *v, float w, float M, const float *r2, float *out)
{
    for (int i = 0; i < n; i++) {
        prr::DevSphere S;
        std::memset(&S, 0, sizeof S);
        S.cx = (float)c[0]; S.cy = (float)c[1]; S.cz = (float)c[2]; S.r = (float)R;
        out[i] = prr::sphere_path<T>(S, p[3 * i], p[3 * i + 1], p[3 * i + 2], v[3 * i], v[3 * i + 1], v[3 * i + 2], w, M, r2[i]);
    }
}
extern "C" void path32(int n, const double *c, double R, const float *p, const float *v, float w, float M, const float *r2, float *out)
{
    each(n, c, R, p, v, w, M, r2, out);
}
extern "C" void path64(int n, const double *c, double R, const double *p, const double *v, float w, float M, const float *r2, float *out)
{
    each(n, c, R, p, v, w, M, r2, out);
}
"""


@pytest.fixture(scope="module")
def lib():
    return library(SOURCE)


def path(lib, c, R, p, v, w, M, r2):
    p, v, c = np.ascontiguousarray(p), np.ascontiguousarray(v, dtype=p.dtype), np.ascontiguousarray(c, dtype=np.float64)
    r2, out = np.ascontiguousarray(r2, dtype=F), np.empty(len(p), dtype=F)
    fn = lib.path32 if p.dtype == F else lib.path64
    q = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    fn(len(p), q(c), C.c_double(R), q(p), q(v), C.c_float(w), C.c_float(M), q(r2), q(out))
    return np.maximum(out.astype(float), 0.0)


def start(rng, n, R, w):
    """Points in and just around the sphere, most rays flying in."""
    rho = unit(rng, n) * (np.sqrt(R * R + w / 3) * rng.uniform(0.02, 1.3, n) ** 0.7)[:, None]
    v = unit(rng, n)
    flip = (rng.random(n) < 0.8) & ((rho * v).sum(1) > 0)
    return rho, np.where(flip[:, None], -v, v)


@pytest.mark.parametrize("w", [1e-4, 1e-6])
@pytest.mark.parametrize("R,far", [(0.01, 30.0), (0.01, 90.0), (0.05, 90.0), (0.2, 90.0), (1.0, 14.0), (0.02, 900.0), (5.0, 900.0)])
def test_no_hit_between_rounded_positions(lib, R, far, w):
    """Straight flight whose points are rounded to FP32, and the test of the reference in FP32 at each of them."""
    rng = np.random.default_rng(7)
    n = 120_000
    c = (unit(rng, 1)[0] * far).astype(F)
    rho, v = start(rng, n, R, w)
    v = v.astype(F)
    x = c.astype(float) + rho
    S = path(lib, c, R, x.astype(F), v, w, 1e-9, np.full(n, far * far))
    assert R * R < 1e-6 * far or (S > 0).mean() > 0.2  # it is of use where the sphere is not lost in the rounding
    for t in np.linspace(0.0, 1.0, 41):
        at = (x + (S * t)[:, None] * v).astype(F)
        d = hit_distance(at - c, v, F(R))
        assert not np.any((S > 0) & (d * d <= F(w)))


def test_no_hit_between_double_positions(lib):
    rng = np.random.default_rng(8)
    n, R, w, c = 120_000, 0.01, 1e-4, np.array([60.0, -60.0, 30.0])
    rho, v = start(rng, n, R, w)
    S = path(lib, c, R, c + rho, v, w, 1e-9, np.full(n, 8100.0))
    assert (S > 0).mean() > 0.5
    for t in np.linspace(0.0, 1.0, 41):
        d = hit_distance(rho + (S * t)[:, None] * v, v, R)
        assert not np.any((S > 0) & (d * d <= w))


@pytest.mark.parametrize("M,R,dist", [(0.2, 5.0, 4.5), (0.05, 3.0, 2.5), (0.5, 5.0, 5.2), (1.0, 5.0, 6.0), (0.1, 2.0, 1.95)])
def test_the_curvature_bound_holds_along_the_whole_path(lib, M, R, dist):
    """Spheres that reach to the hole, rays of every impact parameter from 3 M on: where r falls along the path the curvature grows
    as 1/r^2, and the bound taken at its start has to cover it: with 10 M / r^2 and a factor 1.2^2 for the growth of D^2."""
    rng = np.random.default_rng(9)
    n, w, c = 30_000, 1e-4, np.array([dist, 0.0, 0.0])
    r = 4.0 * M * np.exp(rng.uniform(0.0, 2.5, n))
    x = unit(rng, n) * r[:, None]
    x = x[((x - c) ** 2).sum(1) < R * R]
    n, r = len(x), np.sqrt((x * x).sum(1))
    d = unit(rng, n) * (rng.uniform(3.0, 7.0, n) * M)[:, None] - x
    d /= np.sqrt((d * d).sum(1))[:, None]
    p, pt = null_momentum(d.T, ks(*x.T, M, 0.0))
    s = np.concatenate((x.T, p))
    speed = lambda s: rhs(s, pt, M, 0.0)[:3] / np.sqrt((rhs(s, pt, M, 0.0)[:3] ** 2).sum(0))  # noqa: E731
    S = path(lib, c, R, x, speed(s).T, w, M, r * r)
    assert (S > 0).any()
    kappa, flown, h, D0 = 10.0 * M / (r * r), np.zeros(n), np.full(n, 0.02 * M), np.sqrt(((x - c) ** 2).sum(1))
    while np.any(flown < S):
        y, _ = attempt(s, pt, M, 0.0, h, 1e-9, 1e-9)
        step = np.sqrt(((y[:3] - s[:3]) ** 2).sum(0))
        flown, before, s = flown + step, speed(s), y
        on = flown <= S
        turn = np.sqrt(((speed(s) - before) ** 2).sum(0)) / step
        rho = s[:3].T - c
        dist_hit = hit_distance(rho, speed(s).T, R)
        assert not np.any(on & (dist_hit * dist_hit <= w))
        assert np.all((turn * (rho * rho).sum(1) <= kappa * D0 * D0)[on])
