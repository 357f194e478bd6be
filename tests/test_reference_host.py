"""REFERENCE mode's stepper (parrelray_b200/csrc/ref_stepper.cuh) compiled for the host: leaving out the sixth stage, the
error and the sphere test changes no bit of a ray against the same stepper with nothing left out, a plug-in's geodesic
is called six times an attempt, and the sphere test runs wherever it could pass."""
import ctypes as C

import numpy as np
import pytest

from host_device import library
from parrelray_b200 import abi

SOURCE = r"""
#include "ref_stepper.cuh"
using namespace prr;

struct Plain {  // the built-in hooks with every test and stage evaluated
    static constexpr bool kSpherical = false;
    static constexpr bool kErrorBound = false;
    const FrameParams &fp;
    mutable long long geods = 0;
    void metric(const RefRay &R, float g[16]) const { ref_metric(fp, R, g); }
    V4<float> geod(const V4<float> &x, const V4<float> &u) const
    {
        geods++;
        return fp.metric == PRR_METRIC_KERR ? ref_geod<true>(fp, x, u) : ref_geod<false>(fp, x, u);
    }
    bool loop(RefRay &) const { return true; }
    bool update(RefRay &R, float h) const
    {
        if (intersect_scene<float>(fp, R.r.x, R.r.y, R.r.z, R.u.x, R.u.y, R.u.z, h).hit) { R.result = PRR_RESULT_INTERSECTION; return false; }
        return true;
    }
    bool endloop(RefRay &R, float th) const
    {
        float r = metric_radius<float>(fp, R.r.x, R.r.y, R.r.z);
        if (r >= fp.rout || (fp.metric != PRR_METRIC_FLAT && r <= fp.rstop)) { R.result = PRR_RESULT_SUCCESS; return false; }
        Hit c = intersect_scene<float>(fp, R.r.x, R.r.y, R.r.z, R.u.x, R.u.y, R.u.z, th);
        if (c.hit) { R.u = {c.r, c.g, c.b, 0.0f}; R.result = PRR_RESULT_INTERSECTION; return false; }
        return true;
    }
};

static FrameParams frame(int metric, float M, float a, int w, int h, float incl, float hmax, float eps, int ns, const float *sph)
{
    FrameParams fp;
    std::memset(&fp, 0, sizeof fp);
    fp.width = w; fp.height = h; fp.samples = 1; fp.nsub = 1; fp.vfov = 0.9f;
    fp.cam[0] = 12.0f * std::sin(incl); fp.cam[2] = 12.0f * std::cos(incl);
    fp.alpha = 3.14159274f; fp.beta = incl - 1.57079637f;
    fp.metric = metric; fp.M = M; fp.a = a; fp.rs = 2.0f * M;
    const float rp = metric == PRR_METRIC_KERR ? M + std::sqrt(M * M - a * a) : (metric == PRR_METRIC_FLAT ? 0.0f : fp.rs);
    fp.rstop = rp + 0.01f; fp.rout = 30.0f;
    fp.h = 0.01f; fp.hmin = 1e-3f; fp.hmax = hmax; fp.eps = eps;
    fp.nspheres = ns;
    for (int s = 0; s < ns; s++) {
        const float R = sph[4 * s + 3];
        fp.sph[s].cx = sph[4 * s]; fp.sph[s].cy = sph[4 * s + 1]; fp.sph[s].cz = sph[4 * s + 2]; fp.sph[s].r = R;
        fp.sph[s].far2 = (float)((R * (double)R + hmax / 3.0) * 1.001);  // render.cu:build_plan
    }
    return fp;
}

template <class H> static void trace(const FrameParams &fp, const H &hk, int k, RefRay &R)
{
    ref_init_h(fp, hk, k % fp.width, k / fp.width, 0, R);
    ref_rkf_h(fp, hk, R);
}

// result, accepted, attempts and surplus geodesics of each ray; returns the rays that differ in any bit
extern "C" int compare(int metric, float M, float a, int w, int h, float incl, float hmax, float eps, int ns, const float *sph, int *out)
{
    const FrameParams fp = frame(metric, M, a, w, h, incl, hmax, eps, ns, sph);
    int bad = 0;
    for (int k = 0; k < w * h; k++) {
        RefRay A, B;
        Plain hk{fp};
        if (metric == PRR_METRIC_KERR) trace(fp, BuiltinHooks<true>{fp}, k, A);
        else trace(fp, BuiltinHooks<false>{fp}, k, A);
        trace(fp, hk, k, B);
        bad += std::memcmp(&A.r, &B.r, sizeof A.r) || std::memcmp(&A.u, &B.u, sizeof A.u) || A.result != B.result ||
               A.accepted != B.accepted || A.attempts != B.attempts;
        out[4 * k] = A.result; out[4 * k + 1] = A.accepted; out[4 * k + 2] = A.attempts;
        out[4 * k + 3] = (int)(hk.geods - 6ll * B.attempts);
    }
    return bad;
}

// the sphere test against itself behind ref_near, over given states; returns the states that answer differently
extern "C" int near_differs(int n, const float *x, const float *u, const float *sph, int ns, float hmax, float window)
{
    const FrameParams fp = frame(PRR_METRIC_FLAT, 0.0f, 0.0f, 1, 1, 1.0f, hmax, 1e-3f, ns, sph);
    int bad = 0;
    for (int i = 0; i < n; i++) {
        const V4<float> p = {x[3 * i], x[3 * i + 1], x[3 * i + 2], 0.0f}, v = {u[3 * i], u[3 * i + 1], u[3 * i + 2], 1.0f};
        const bool hit = intersect_scene<float>(fp, p.x, p.y, p.z, v.x, v.y, v.z, window).hit;
        bad += hit && !ref_near(fp, p);
    }
    return bad;
}
extern "C" int finite_stage(float M, const float *x, const float *u, float h)
{
    const FrameParams fp = frame(PRR_METRIC_SCHWARZSCHILD, M, 0.0f, 1, 1, 1.0f, 0.1f, 1e-3f, 0, nullptr);
    return ref_finite_stage(fp, {x[0], x[1], x[2], 0.0f}, {u[0], u[1], u[2], 1.0f}, h);
}
"""
SPHERES = {"none": [], "ring": [(6.0, 0.0, 0.0, 1.0), (-4.0, 5.0, 0.5, 0.7)], "near": [(2.5, 1.5, 0.0, 1.5), (3.0, -3.0, 1.0, 0.05)]}


@pytest.fixture(scope="module")
def lib():
    return library(SOURCE)


def fp(a):
    return a.ctypes.data_as(C.c_void_p)


@pytest.mark.parametrize("eps,hmax", [(1e-3, 0.1), (1e-2, 0.5), (1e-4, 0.1)])
@pytest.mark.parametrize("spheres", sorted(SPHERES))
@pytest.mark.parametrize("metric,M,a", [(abi.METRIC_KERR, 1.0, 0.9), (abi.METRIC_SCHWARZSCHILD, 1.0, 0.0), (abi.METRIC_SCHWARZSCHILD, 0.0, 0.0),
                                        (abi.METRIC_FLAT, 0.0, 0.0)])
def test_nothing_left_out_matters(lib, metric, M, a, spheres, eps, hmax):
    """An odd frame on the equator: rays with exact zeros among them."""
    w, h = 9, 5
    s = np.array(SPHERES[spheres], dtype=np.float32).reshape(-1, 4)
    out = np.zeros((w * h, 4), dtype=np.int32)
    f = C.c_float
    bad = lib.compare(metric, f(M), f(a), w, h, f(1.57079637), f(hmax), f(eps), len(s), fp(s), fp(out))
    assert bad == 0
    assert (out[:, 3] == 0).all()  # six evaluations of an unknown geodesic in every attempt
    assert (out[:, 1] > 10).any()
    if spheres == "ring":
        assert (out[:, 0] == abi.RESULT_INTERSECTION).any()


def test_no_hit_is_lost_on_states_that_are_not_finite(lib):
    rng = np.random.default_rng(3)
    n = 20_000
    s = np.array(SPHERES["ring"], dtype=np.float32)
    odd = np.array([0.0, -0.0, 1e-25, 1e-20, 1e-15, 1.0, 1e10, 1e15, 1e18, 1e20, 3e38, np.inf, np.nan], dtype=np.float32)
    x = rng.normal(size=(n, 3)).astype(np.float32) * 8
    u = rng.normal(size=(n, 3)).astype(np.float32)
    with np.errstate(over="ignore", invalid="ignore"):
        u = np.where(rng.random((n, 1)) < 0.5, u * rng.choice(odd, (n, 1)), np.where(rng.random((n, 3)) < 0.4, rng.choice(odd, (n, 3)), u))
        x = np.where(rng.random((n, 3)) < 0.2, x * rng.choice(odd, (n, 3)), x)
    x, u = np.ascontiguousarray(x, dtype=np.float32), np.ascontiguousarray(u, dtype=np.float32)
    for window in (1e-4, 0.1):
        assert lib.near_differs(n, fp(x), fp(u), fp(s), len(s), C.c_float(0.1), C.c_float(window)) == 0


def test_stages_outside_the_tame_range_are_evaluated(lib):
    call = lambda M, x, u, h: lib.finite_stage(C.c_float(M), fp(np.array(x, np.float32)), fp(np.array(u, np.float32)), C.c_float(h))  # noqa: E731
    assert call(1.0, (8, 0, 0), (-1, 0, 0), 1e-4) == 1
    for x, u, h in [((3, 0, 0), (-1, 0, 0), 1e-4), ((8, 0, 0), (np.nan, 0, 0), 1e-4), ((8, 0, 0), (np.inf, 0, 0), 1e-4),
                    ((8, 0, 0), (1e6, 0, 0), 1e-12), ((1e9, 0, 0), (1, 0, 0), 1e-4), ((np.nan, 0, 0), (1, 0, 0), 1e-4),
                    ((8, 0, 0), (-1, 0, 0), 0.1), ((8, 0, 0), (-1, 0, 0), 0.5), ((np.inf, 0, 0), (1, 0, 0), 1e-4)]:
        assert call(1.0, x, u, h) == 0
    assert call(0.0, (1e-6, 0, 0), (1, 0, 0), 1e-10) == 0
