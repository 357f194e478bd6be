"""Where REFERENCE mode leaves the sixth stage and the error out (parrelray_b200/csrc/ref_stepper.cuh,
ref_small_error), restated in numpy: over random states, masses and spins that satisfy the rule, the embedded
difference of the mode's own stages (velocity inputs h u where h du belongs) is under the bound, and in FP32, summed
as the mode sums it, under the eps^0.2 step control's 0.9^5 of eps.

Pure mathematics: no GPU, no oracle.
"""
import numpy as np
import pytest

from test_error_skip import A, B4, B5
from test_geod_closed_form import geod


def accel(x, u, M, a):
    """test_geod_closed_form.geod over columns, in the precision of x."""
    T = x.dtype
    X, Y, Z = x[0], x[1], x[2]
    hb = (X * X + Y * Y + Z * Z - a * a) / 2
    Sh = np.sqrt(hb * hb + a * a * Z * Z)
    r2 = hb + Sh
    r, iS, iq = np.sqrt(r2), 1 / (2 * Sh), 1 / (r2 + a * a)
    lz = Z / r
    al, be = r * iS, a * lz * iS
    lx, ly = (r * X + a * Y) * iq, (r * Y - a * X) * iq
    ka, ta = al * (al * al - 3 * be * be), be * (3 * al * al - be * be)
    lu = lx * u[0] + ly * u[1] + lz * u[2]
    L, N = lu + u[3], u[0] * u[0] + u[1] * u[1] + u[2] * u[2] - lu * lu
    B = L * (-ka * (X * u[0] + Y * u[1] + Z * u[2]) - a * ta * u[2]) + al * al * N - M * al * L * L * (al * al - be * be)
    c, h = 2 * al * be * L, L * L / 2
    return (2 * M * np.stack((c * (ly * u[2] - lz * u[1]) - B * lx - h * ka * X, c * (lz * u[0] - lx * u[2]) - B * ly - h * ka * Y,
                              c * (lx * u[1] - ly * u[0]) - B * lz - h * ka * Z - h * a * ta, B))).astype(T)


def difference(x, u, M, a, h):
    """max |y5 - y4| of one attempt, each solution summed left to right as the source spells it."""
    T = x.dtype.type
    kx, ku = [h * u], [h * accel(x, u, M, a)]
    for i in range(1, 6):
        zx, zu = x, u + T(A[i][0]) * kx[0]
        for j in range(i):
            zx = zx + T(A[i][j]) * kx[j]
        for j in range(1, i):
            zu = zu + T(A[i][j]) * ku[j]
        kx.append(h * zu)
        ku.append(h * accel(zx, zu, M, a))
    out = []
    for y, k in ((x, kx), (u, ku)):
        s4 = s5 = y
        for c4, c5, kk in zip(B4, B5, k):
            s4, s5 = s4 + T(c4) * kk, s5 + T(c5) * kk
        out.append(np.abs(s5 - s4).max(0))
    return np.maximum(*out)


def sample(rng, n, M):
    a = M * rng.uniform(-1, 1, n)
    U = np.exp(rng.uniform(np.log(0.3), np.log(4.0), n))
    r = (4.02 * M if M else 0.5) * np.exp(rng.uniform(0, 3.0, n))
    ct, ph = rng.uniform(-1, 1, n), rng.uniform(0, 2 * np.pi, n)
    st = np.sqrt(1 - ct * ct)
    R = np.sqrt(r * r + a * a)
    x = np.stack((R * st * np.cos(ph), R * st * np.sin(ph), r * ct, rng.uniform(0, 100, n)))
    u = rng.normal(size=(4, n))
    u *= U / np.abs(u).max(0)
    h = np.minimum(0.25, rng.uniform(0.05, 1.0, n) * r / (16 * U))
    return x, u, a, h, r, U


@pytest.mark.parametrize("M", [0.0, 0.05, 0.3, 1.0, 3.0])
def test_difference_is_under_the_bound(M):
    x, u, a, h, r, U = sample(np.random.default_rng(4), 150_000, M)
    bound = h * U * (0.01 * h + 0.2 * (h * U / r) * M / r)
    noise = 1e-14 * (np.abs(x).max(0) + U)
    assert (difference(x, u, M, a, h) <= bound + noise).all()


@pytest.mark.parametrize("M,eps", [(1.0, 1e-3), (0.3, 1e-3), (1.0, 3e-4), (0.0, 1e-3)])
def test_fp32_difference_keeps_the_step_at_hmax(M, eps):
    x, u, a, h, r, U = sample(np.random.default_rng(5), 150_000, M)
    X = np.sqrt((x[:3] ** 2).sum(0)) + np.abs(x[3]) + U
    ok = h * U * (0.01 * h + 0.2 * (h * U / r) * M / r) + 7.2e-7 * X <= 0.5 * eps
    assert ok.any()
    f = lambda v: np.asarray(v, dtype=np.float32)  # noqa: E731
    d = difference(f(x[:, ok]), f(u[:, ok]), f(M), f(a[ok]), f(h[ok]))
    assert d.max() < 0.9**5 * eps


def test_the_columns_form_is_the_closed_form():
    rng = np.random.default_rng(6)
    x, u = rng.normal(size=(4, 20)) * 9, rng.normal(size=(4, 20))
    got = accel(x, u, 1.1, 0.7)
    for k in range(20):
        assert np.allclose(got[:, k], geod(x[:3, k], u[:, k], 1.1, 0.7), rtol=1e-12, atol=1e-14)
