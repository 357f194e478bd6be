"""The Hamiltonian renderer's quick accept step (parrelray_b200/csrc/k_ham.cu: ham_quick_accept, sphere_path,
ham_run_limit): what it may skip is skipped only where it cannot matter.

CPU: the far radius R^2 + w/3 of Sphere::intersects, and the path lengths of sphere_path, restated in numpy FP32 and
checked against the exact test along curved paths.  GPU: the caps that a run of quick steps must stop at, against a
numpy integrator that looks at every step.
"""
import numpy as np
import pytest

from parrelray_b200 import abi
from test_error_skip import test_fp64_rays_take_the_steps_of_a_full_estimator as take_the_steps

F = np.float32


def hit_distance(rho, v, R):
    """Sphere::intersects' distance along the unit vector v from rho (relative to the centre); nan: missed."""
    dvp = (rho * v).sum(-1)
    disc = dvp * dvp - ((rho * rho).sum(-1) - R * R)
    with np.errstate(invalid="ignore"):
        d = -2.0 * dvp - np.sqrt(disc)
    return np.where(d >= 0.0, d, np.nan)


def unit(rng, n):
    v = rng.normal(size=(n, 3))
    return v / np.linalg.norm(v, axis=1, keepdims=True)


@pytest.mark.parametrize("w", [1e-4, 0.1, 1.0])
def test_no_hit_outside_the_far_radius(w):
    rng = np.random.default_rng(2)
    n = 400_000
    R = np.exp(rng.uniform(np.log(0.05), np.log(5.0), n))
    D = np.sqrt(R * R + w / 3) * np.where(rng.random(n) < 0.5, 1.0 + 1e-9, rng.uniform(1.0, 3.0, n))
    v = unit(rng, n)
    # directions near the minimum of d over b as well as random ones: b^2 = 4c/3
    c = D * D - R * R
    b = np.where(rng.random(n) < 0.5, np.minimum(np.sqrt(4 * c / 3) * rng.uniform(0.98, 1.02, n), D), rng.uniform(-1, 1, n) * D)
    perp = np.cross(v, unit(rng, n))
    perp /= np.linalg.norm(perp, axis=1, keepdims=True)
    rho = -b[:, None] * v + np.sqrt(np.maximum(D * D - b * b, 0.0))[:, None] * perp
    d = hit_distance(rho, v, R)
    assert not np.any(d * d <= w * (1 - 1e-6))


def sphere_path(rho, v, R, w, M, r2):
    """k_ham.cu's sphere_path, every operation in FP32."""
    rho, v, R, w, M, r2 = (np.asarray(x, dtype=F) for x in (rho, v, R, w, M, r2))
    D2 = np.maximum((rho * rho).sum(-1, dtype=F), F(1e-30))
    D, sqw = np.sqrt(D2), np.sqrt(w)
    away = F(0.9) * (D - F(1.1) * R - sqw)
    b = -(v * rho).sum(-1, dtype=F)
    disc = b * b - (D2 - R * R)
    kap = F(10) * M / r2
    grow, err = F(2) * D2 * kap, F(4e-6) * D2
    sw = F(1.00001) * sqw + F(1e-5) * D
    p = np.maximum(disc, F(0))
    S1 = np.minimum(F(0.25) * (F(2) * b - np.sqrt(p + err) - sw), F(0.2) * D)
    ok1 = (S1 > 0) & (F(2) * (b - S1 * (F(1) + D * kap)) - np.sqrt(np.maximum(p + grow * S1 + err, F(0))) > sw)
    S2 = F(0.05) * D
    ok2 = (disc + grow * S2 + err < 0) | (F(2) * (b + D * kap * S2) - np.sqrt(np.maximum(disc - grow * S2 - err, F(0))) < F(-1e-5) * D)
    S = np.where(ok1, S1, np.where(ok2, S2, F(0)))
    return np.where(away > 0, away, np.where(r2 >= F(16) * M * M, S, F(0)))


@pytest.mark.parametrize("R,r", [(0.5, 6.5), (1.2, 14.0), (2.0, 5.0), (0.05, 9.0)])
def test_no_hit_within_the_path_length(R, r):
    """Arcs of the largest curvature (4 M / r^2) in random planes from points in and around the sphere: the exact test
    with the window hmin never passes before the length that sphere_path gives."""
    rng = np.random.default_rng(3)
    n, w, M = 60_000, 1e-4, 1.0
    rho = unit(rng, n) * (R * rng.uniform(0.02, 1.3, n) ** 0.7)[:, None]
    v = unit(rng, n)
    aim = rng.random(n) < 0.6  # flying in
    v = np.where((aim & ((rho * v).sum(1) > 0))[:, None], -v, v)
    side = np.cross(v, unit(rng, n))
    side /= np.linalg.norm(side, axis=1, keepdims=True)
    S = sphere_path(rho, v, R, w, M, r * r).astype(float)
    assert (S > 0).mean() > 0.5
    k = 4.0 * M / (r * r)
    for t in np.linspace(0.0, 1.0, 41):
        s = S * t
        x = rho + (np.sin(k * s) / k)[:, None] * v + ((1 - np.cos(k * s)) / k)[:, None] * side
        u = np.cos(k * s)[:, None] * v + np.sin(k * s)[:, None] * side
        d = hit_distance(x, u, R)
        assert not np.any((S > 0) & (d * d <= w))


@pytest.mark.gpu
@pytest.mark.parametrize("kw", [
    dict(r=20.0, spin=0.8, max_steps=3), dict(r=20.0, spin=0.8, max_steps=66), dict(r=20.0, spin=0.8, max_steps=1000),
    dict(r=30.0, spin=0.4, hmax=0.6, rout=4000.0), dict(r=12.0, spin=0.9, horizon_eps=6.0), dict(r=25.0, spin=0.2, rout=25.5)])
def test_quick_runs_stop_at_the_caps(gpu, kw):
    """max_steps, the loop bound l < 1000, a stop radius outside the cruise radius, an escape at once."""
    take_the_steps(gpu, kw)
