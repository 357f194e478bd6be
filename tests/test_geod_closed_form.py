"""The closed forms of the Kerr-Schild geodesic and its vector-Jacobian product that the adjoint's reverse sweep
uses (parrelray_b200/csrc/geod_vjp.cuh), restated in numpy operation by operation: the acceleration against the
contraction of Gamma u u from numerical Christoffel symbols, the product against central differences.

Pure mathematics: no GPU, no oracle.
"""
import numpy as np
import pytest


def metric(x, M, a):
    X, Y, Z = x
    hb = 0.5 * (X * X + Y * Y + Z * Z - a * a)
    r2 = hb + np.sqrt(hb * hb + a * a * Z * Z)
    r = np.sqrt(r2)
    q = r2 + a * a
    l = np.array([(r * X + a * Y) / q, (r * Y - a * X) / q, Z / r, 1.0])
    return np.diag([1.0, 1.0, 1.0, -1.0]) + 2 * M * r * r2 / (r2 * r2 + a * a * Z * Z) * np.outer(l, l)


def contraction(x, u, M, a, h=1e-4):
    """-Gamma^k_mn u^m u^n with fourth-order differences of the metric (static: d_t = 0)."""
    dg = np.zeros((4, 4, 4))
    for k in range(3):
        e = np.zeros(3)
        e[k] = h
        dg[k] = (8 * (metric(x + e, M, a) - metric(x - e, M, a)) - (metric(x + 2 * e, M, a) - metric(x - 2 * e, M, a))) / (12 * h)
    low = np.einsum("kmn,k,n->m", dg, u, u) - 0.5 * np.einsum("mkn,k,n->m", dg, u, u)
    return -np.linalg.solve(metric(x, M, a), low)


def point(x, a):
    X, Y, Z = x
    hb = 0.5 * (X * X + Y * Y + Z * Z - a * a)
    Sh = np.sqrt(hb * hb + a * a * Z * Z)
    r2 = hb + Sh
    r, iS, iq = np.sqrt(r2), 0.5 / Sh, 1 / (r2 + a * a)
    lz = Z / r
    al, be = r * iS, a * lz * iS
    l = np.array([(r * X + a * Y) * iq, (r * Y - a * X) * iq, lz])
    return r, iq, al, be, l, al * (al * al - 3 * be * be), be * (3 * al * al - be * be)


def geod(x, u, M, a):
    _, _, al, be, l, ka, ta = point(x, a)
    us, L = u[:3], l @ u[:3] + u[3]
    N = us @ us - (l @ us) ** 2
    du = -ka * (x @ us) - a * ta * us[2]
    B = L * du + al * al * N - M * al * L * L * (al * al - be * be)
    s = 2 * al * be * L * np.cross(l, us) - B * l - 0.5 * L * L * (ka * x + np.array([0, 0, a * ta]))
    return 2 * M * np.append(s, B)


def vjp(x, u, M, a, w):
    r, iq, al, be, l, ka, ta = point(x, a)
    us, ws, (X, Y, Z) = u[:3], w[:3], x
    ab, g, at = al * be, al * al - be * be, a * ta
    L, om, c = l @ us + u[3], l @ ws - w[3], np.cross(us, ws)
    T, h, lu = l @ c, 0.5 * L * L, l @ us
    xu, xw, N = x @ us, x @ ws, us @ us - lu * lu
    du, dw = -ka * xu - at * us[2], -ka * xw - at * ws[2]
    B = L * du + al * al * N - M * al * L * L * g
    psi = h * dw + 2 * ab * L * T - om * B
    P_du, P_N = -om * L, -om * al * al
    P_L = 2 * ab * T + L * dw - om * (du - 2 * M * al * L * g)
    P_lu = P_L - 2 * P_N * lu
    P_ka, qz = -(P_du * xu + h * xw), P_du * us[2] + h * ws[2]
    P_al = 2 * be * L * T - om * (2 * al * N - M * L * L * (g + 2 * al * al)) + 3 * g * P_ka - 6 * ab * a * qz
    P_be = 2 * al * L * T - 2 * om * be * M * al * L * L - 6 * ab * P_ka - 3 * g * a * qz
    v = P_lu * us - B * ws + 2 * ab * L * c
    gx = (al * (v - l * (l @ v)) - be * np.cross(v, l) - (ka * P_al + ta * P_be) * x - ka * (P_du * us + h * ws)
          + np.array([0, 0, a * (ka * P_be - ta * P_al)]))
    gu = P_lu * l + 2 * P_N * us + 2 * ab * L * np.cross(ws, l) - ka * P_du * x - np.array([0, 0, at * P_du])
    ra = Z * be - a * al
    k2 = 2 * (r * ra + a)
    la = np.array([(ra * X + Y - l[0] * k2) * iq, (ra * Y - X - l[1] * k2) * iq, -l[2] * ra / r])
    ga = P_al * (ka * a - ta * Z) + P_be * (ka * Z + at) + v @ la - ta * qz
    return 2 * M * gx, 2 * M * np.append(gu, P_L), 2 * (psi + om * M * al * L * L * g), 2 * M * ga


def states(n=40, seed=0):
    rng = np.random.default_rng(seed)
    for _ in range(n):
        x = rng.normal(size=3)
        x *= rng.uniform(2.5, 40.0) / np.linalg.norm(x)
        yield x, rng.normal(size=4), rng.normal(size=4)


@pytest.mark.parametrize("M,a", [(1.0, 0.0), (1.0, 0.95), (1.3, -1.2), (0.4, 0.4)])
def test_acceleration_is_the_christoffel_contraction(M, a):
    for x, u, _ in states():
        ref = contraction(x, u, M, a)
        # fourth-order differences, h = 1e-4: rounding 1e-12 of the metric over h
        assert np.abs(geod(x, u, M, a) - ref).max() <= 1e-9 * (1 + np.abs(u).max() ** 2)


@pytest.mark.parametrize("M,a", [(1.0, 0.0), (1.0, 0.95), (1.3, -1.2), (0.0, 0.0)])
def test_product_is_the_derivative(M, a):
    d = 1e-5
    for x, u, w in states(seed=1):
        gx, gu, gM, ga = vjp(x, u, M, a, w)
        f = lambda x_, u_, M_, a_: w @ geod(x_, u_, M_, a_)  # noqa: E731
        num = [(f(x + d * e, u, M, a) - f(x - d * e, u, M, a)) / (2 * d) for e in np.eye(3)]
        num += [(f(x, u + d * e, M, a) - f(x, u - d * e, M, a)) / (2 * d) for e in np.eye(4)]
        num += [(f(x, u, M + d, a) - f(x, u, M - d, a)) / (2 * d), (f(x, u, M, a + d) - f(x, u, M, a - d)) / (2 * d)]
        got = np.concatenate([gx, gu, [gM, ga]])
        assert np.abs(got - num).max() <= 1e-8 * (1 + np.abs(got).max())
