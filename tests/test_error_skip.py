"""Where the Hamiltonian renderer leaves the error estimate out (parrelray_b200/csrc/k_ham.cu,
ham_cruise_r2), restated in numpy.

CPU: over random null states at or outside the radius the rule returns, in FP64 and with every
operation rounded to FP32, the scaled error of a step of hmax stays under 0.9^5 (where the step control
0.9 h err^(-1/5) leaves hmax), so the full evaluation would decide the same.
GPU: FP64 rays take the steps of a numpy integrator that always evaluates the error.
"""
import math

import numpy as np
import pytest

from parrelray_b200 import abi, scenes

A = [[], [1 / 4], [3 / 32, 9 / 32], [1932 / 2197, -7200 / 2197, 7296 / 2197], [439 / 216, -8.0, 3680 / 513, -845 / 4104],
     [-8 / 27, 2.0, -3544 / 2565, 1859 / 4104, -11 / 40]]
B4 = [25 / 216, 0.0, 1408 / 2565, 2197 / 4104, -1 / 5, 0.0]
B5 = [16 / 135, 0.0, 6656 / 12825, 28561 / 56430, -9 / 50, 2 / 55]


def ks(x, y, z, M, a):
    hb = 0.5 * (x * x + y * y + z * z - a * a)
    r2 = hb + np.sqrt(hb * hb + a * a * z * z)
    r = np.sqrt(r2)
    q = r2 + a * a
    return r, 2 * M * r * r2 / (r2 * r2 + a * a * z * z), ((r * x + a * y) / q, (r * y - a * x) / q, z / r)


def rhs(s, pt, M, a):
    """In the precision of s (numpy keeps float32 operands in float32)."""
    x, y, z, px, py, pz = s
    a2 = a * a
    half, two = s.dtype.type(0.5), s.dtype.type(2)
    hb = half * (x * x + y * y + z * z - a2)
    Sh = np.sqrt(hb * hb + a2 * z * z)
    r2 = hb + Sh
    r = np.sqrt(r2)
    q, Sig = r2 + a2, r2 * r2 + a2 * z * z
    rx, ry, rz = x * r / (two * Sh), y * r / (two * Sh), z * q / (two * Sh * r)
    f = two * M * r * r2 / Sig
    c1 = f * (s.dtype.type(3) / r - s.dtype.type(4) * r * r2 / Sig)
    lx, ly, lz = (r * x + a * y) / q, (r * y - a * x) / q, z / r
    lp = lx * px + ly * py
    Lam = lp + lz * pz - pt
    Pp = (x * px + y * py - two * r * lp) / q - pz * lz / r
    h2, fL = half * Lam * Lam, f * Lam
    return np.stack((px - fL * lx, py - fL * ly, pz - fL * lz, h2 * c1 * rx + fL * (rx * Pp + (r * px - a * py) / q),
                     h2 * c1 * ry + fL * (ry * Pp + (a * px + r * py) / q),
                     h2 * (c1 * rz - two * f * a2 * z / Sig) + fL * (rz * Pp + pz / r)))


def attempt(s, pt, M, a, h, rtol, atol):
    """4th-order solution and scaled error of one attempt."""
    T = s.dtype.type
    k = []
    for row in A:
        z = s
        for c, kk in zip(row, k):
            z = z + T(c) * kk
        k.append(h * rhs(z, pt, M, a))
    y = s + sum(T(c) * kk for c, kk in zip(B4, k) if c)
    e = sum(T(c5 - c4) * kk for c5, c4, kk in zip(B5, B4, k) if c5 != c4)
    return y, (np.abs(e) / (T(atol) + T(rtol) * np.maximum(np.abs(s), np.abs(y)))).max(axis=0)


def null_momentum(d, r_f_l):
    """Covariant momentum of the future null vector (d, u^t), |d| = 1."""
    _, f, l = r_f_l
    ld = l[0] * d[0] + l[1] * d[1] + l[2] * d[2]
    qa, qb, qc = f - 1, 2 * f * ld, 1 + f * ld * ld
    rt = np.sqrt(qb * qb - 4 * qa * qc)
    ut = np.maximum((-qb + rt) / (2 * qa), (-qb - rt) / (2 * qa))
    Lu = ld + ut
    return np.stack([d[k] + f * l[k] * Lu for k in range(3)]), -ut + f * Lu


def rule_radius(M, E, hmax, atol, noise):
    """ham_cruise_r2 without the a^2 of the Euclidean test; inf where the rule refuses."""
    hE = hmax * E
    h5 = hE**5 / (0.25 * atol)
    r = np.maximum(np.maximum(4 * M, 8 * hE), np.maximum((4 * M * h5) ** 0.2, (7 * M * E * h5) ** (1 / 6)))
    return np.where(noise * hE <= 0.3 * atol, r, np.inf)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("tol,hmax,M", [(1e-6, 0.1, 1.0), (1e-7, 0.1, 1.0), (1e-7, 0.05, 0.2), (1e-5, 0.5, 2.0),
                                        (1e-9, 0.1, 1.0), (1e-6, 0.2, 0.0)])
def test_scaled_error_stays_under_the_step_control(dtype, tol, hmax, M):
    rng = np.random.default_rng(11)
    n = 40_000
    noise = 2.5e-7 if dtype is np.float32 else 5e-16
    a = M * rng.uniform(0.0, 1.0, n) * rng.choice([-1.0, 1.0], n)
    d = rng.normal(size=(3, n))
    d /= np.sqrt((d * d).sum(0))
    lo = rule_radius(M, 1.0, hmax, tol, noise)
    if not np.isfinite(lo):
        pytest.skip("the rule refuses: FP32 rounding is not under this tolerance")
    lo = max(float(lo), 1e-3)
    r = np.where(np.arange(n) % 2 == 0, lo * rng.uniform(1.0, 1.2, n), np.exp(rng.uniform(np.log(lo), np.log(40 * lo), n)))
    ct, ph = rng.uniform(-1, 1, n), rng.uniform(0, 2 * np.pi, n)
    st = np.sqrt(1 - ct * ct)
    x = np.stack((np.sqrt(r * r + a * a) * st * np.cos(ph), np.sqrt(r * r + a * a) * st * np.sin(ph), r * ct))
    p, pt = null_momentum(d, ks(*x, M, a))
    E = np.abs(pt)
    p, pt = p / E, pt / E  # E = 1: hE = hmax
    s = np.concatenate((x, p)).astype(dtype)
    c = lambda v: np.asarray(v, dtype=dtype)  # noqa: E731
    _, err = attempt(s, c(pt), c(M), c(a), c(hmax), tol, tol)
    assert np.isfinite(err).all()
    assert err.max() < 0.9**5


@pytest.mark.gpu
@pytest.mark.parametrize("kw", [
    dict(r=25.0, spin=0.9), dict(r=5.0, spin=0.998), dict(r=30.0, spin=0.0, metric=abi.METRIC_SCHWARZSCHILD),
    dict(r=12.0, spin=0.3, tol=1e-9), dict(r=20.0, spin=1.4, mass=2.0, hmax=1.5, h=0.02), dict(r=9.0, spin=0.0, metric=abi.METRIC_FLAT),
    dict(r=20.0, spin=0.5, hmin=0.1, hmax=0.1), dict(r=6.0, spin=0.7, hmax=40.0, tol=1e-5)])
def test_fp64_rays_take_the_steps_of_a_full_estimator(gpu, kw):
    """Accepted-step counts equal for every ray but the few whose orbit amplifies the FP32 rounding of the ray
    directions (2 %): a decision changed by a skipped estimate would change the counts of whole image regions.
    (Positions are not compared: the same rounding, times the distance and the deflection's derivative, is in them.)"""
    kw = dict(dict(incl_deg=70.0, fov_deg=50.0, metric=abi.METRIC_KERR, precision=abi.PREC_FP64, background=False, tol=1e-6), **kw)
    f = scenes.make_frame(23, 13, **kw)
    state, _, stats = gpu.trace_rays_f64(f)
    M = 0.0 if f.metric == abi.METRIC_FLAT else f.mass
    a = f.spin if f.metric == abi.METRIC_KERR else 0.0
    n = f.nrays
    j = np.arange(n)
    uvx, uvy = state[:, 0], state[:, 1]
    mu = ((0.5 - uvx) * f.width / f.height * f.vfov)
    nu = (0.5 - uvy) * f.vfov
    cb = np.cos(f.cam_beta + nu)
    d = np.stack((cb * np.cos(f.cam_alpha + mu), cb * np.sin(f.cam_alpha + mu), np.sin(f.cam_beta + nu)))
    pos = np.stack([np.full(n, f.cam_pos[k]) for k in range(3)])
    p, pt = null_momentum(d, ks(*pos, M, a))
    s = np.concatenate((pos, p))
    rstop = (M + math.sqrt(M * M - a * a) if M else 0.0) + f.horizon_eps
    h, path, acc = np.full(n, float(f.h)), np.zeros(n), np.zeros(n, int)
    count = np.zeros(n, int)
    while len(j):
        y, err = attempt(s, pt, M, a, h, f.rtol, f.atol)
        with np.errstate(divide="ignore"):
            hn = np.clip(0.9 * h * err**-0.2, f.hmin, f.hmax)
        ok = ~((err > 1) & (h != f.hmin))
        s = np.where(ok, y, s)
        acc = acc + ok
        h = hn
        r = ks(s[0], s[1], s[2], M, a)[0]
        path = np.where(ok, path + h, path)
        done = ok & ((r >= f.rout) | ((r <= rstop) if M else False) | (path >= 1000.0) | (acc >= f.max_steps))
        count[j[done]] = acc[done]
        k = ~done
        s, pt, h, path, acc, j = s[:, k], pt[k], h[k], path[k], acc[k], j[k]
    same = count == state[:, 11]
    assert same.mean() >= 0.98, (same.mean(), stats.as_dict())


@pytest.mark.parametrize("tol,hmax,M", [(1e-6, 0.1, 1.0), (1e-8, 0.05, 0.2), (1e-5, 0.5, 2.0)])
def test_velocity_form_stays_under_the_step_control_too(tol, hmax, M):
    """The (x, u) form of the adjoint's FP64 steps (phys_stepper.cuh, cruise_radius) under the same radius."""
    from test_reference_error_skip import accel

    rng = np.random.default_rng(13)
    n = 40_000
    a = M * rng.uniform(0.0, 1.0, n) * rng.choice([-1.0, 1.0], n)
    d = rng.normal(size=(3, n))
    d /= np.sqrt((d * d).sum(0))
    lo = float(rule_radius(M, 1.0, hmax, tol, 5e-16))
    r = lo * np.exp(rng.uniform(0.0, 3.5, n) * (np.arange(n) % 2))
    ct, ph = rng.uniform(-1, 1, n), rng.uniform(0, 2 * np.pi, n)
    st, R = np.sqrt(1 - ct * ct), np.sqrt(r * r + a * a)
    x = np.stack((R * st * np.cos(ph), R * st * np.sin(ph), r * ct))
    _, f, l = ks(*x, M, a)
    ld = (np.stack(l) * d).sum(0)
    rt = np.sqrt(4 * f * f * ld * ld - 4 * (f - 1) * (1 + f * ld * ld))
    ut = np.maximum((-2 * f * ld + rt) / (2 * (f - 1)), (-2 * f * ld - rt) / (2 * (f - 1)))
    u = np.concatenate((d, ut[None])) / (ut - f * (ld + ut))  # E = 1
    y = np.concatenate((x, np.zeros((1, n)), u))
    k = []
    for row in A:
        z = y + sum((c * kk for c, kk in zip(row, k)), 0 * y)
        k.append(hmax * np.concatenate((z[4:], accel(z[:4], z[4:], M, a))))
    e = sum((c5 - c4) * kk for c5, c4, kk in zip(B5, B4, k))
    assert (np.abs(e) / tol).max() < 0.9**5
