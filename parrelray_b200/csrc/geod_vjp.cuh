// geod_vjp.cuh - the Kerr-Schild geodesic acceleration G = du/dlambda and its
// reverse-mode derivative (vector-Jacobian product) in FP64, in closed form:
// given weights w[4] on the outputs, geod_vjp gives
//   gx[k] = sum_r w_r dG_r/dx_k, gu[k] = sum_r w_r dG_r/du_k (k = x, y, z, t),
//   gM = sum_r w_r dG_r/dM,      ga = sum_r w_r dG_r/da.
// The adjoint of one stage of the RKF45 step needs exactly this product.
//
// With the complex radius R = r + i a cos(theta), R^2 = x^2 + y^2 + (z + i a)^2,
// and 1/R = alpha - i beta, the metric function is f = 2M alpha, and the null
// congruence l is geodesic and shear-free:
//   d_k l_m = alpha (delta_km - l_k l_m) - beta eps_kmn l_n,
// so (l.grad) l = 0 and J l = 0 for J = grad l.  With L = l.u + u^t,
// N = |u|^2 - (l.u)^2, gamma = alpha^2 - beta^2 and 1/R^3 = kappa - i tau,
//   grad alpha = -kappa x - a tau e_z,  grad beta = -tau x + a kappa e_z,
//   B = L (u.grad alpha) + alpha^2 N - M alpha L^2 gamma,
//   G_s = 2M (-B l + 2 alpha beta L (l x u) + 1/2 L^2 grad alpha),  G_t = 2M B
// (geod_ks contracts the Christoffel symbols term by term instead; the two
// agree to rounding).  The product is then the gradient of one scalar,
//   w.G = 2M Psi,  Psi = -omega B + 2 alpha beta L T + 1/2 L^2 (w.grad alpha),
// omega = l.w - w_t, T = l.(u x w), which is differentiated through alpha,
// beta and l.  Both functions leave the factor 2M of G, gx, gu and ga to the
// caller (gM is whole), who has the step length to multiply by as well.
//
// About 100 and 220 FP64 operations, where the contraction and its reverse
// sweep took 130 and 385: one gradient of a 512x512 frame took 59 ms in
// k_adjoint with those, and 39 ms with these.  The time coordinate x^t does
// not enter the acceleration, so gx[3] = 0.
#pragma once
#include "prr_device.cuh"

namespace prr {

// l, alpha, beta, kappa, tau and the reciprocals they come from, at p.
struct KsPoint {
    double r, ir, iq, al, be, lx, ly, lz, a2, b2, ka, ta;
};

PRR_DEV KsPoint ks_point(const V4<double> &p, double a)
{
    KsPoint k;
    const double X = p.x, Y = p.y, Z = p.z, aa = a * a;
    const double hb = 0.5 * (X * X + Y * Y + Z * Z - aa);  // Re(R^2)/2
    const double S2h = hb * hb + aa * Z * Z, iSh = h3_rsqrt(S2h), r2 = S2h * iSh + hb;
    k.ir = h3_rsqrt(r2);
    k.r = r2 * k.ir;
    k.iq = h3_rcp(r2 + aa);
    const double iS = 0.5 * iSh;  // 1/|R|^2
    k.lz = Z * k.ir;
    k.lx = (k.r * X + a * Y) * k.iq;
    k.ly = (k.r * Y - a * X) * k.iq;
    k.al = k.r * iS;
    k.be = a * k.lz * iS;
    k.a2 = k.al * k.al;
    k.b2 = k.be * k.be;
    k.ka = k.al * (k.a2 - 3.0 * k.b2);
    k.ta = k.be * (3.0 * k.a2 - k.b2);
    return k;
}

// G / (2M)
PRR_DEV V4<double> geod_unit(const V4<double> &p, const V4<double> &u, double M, double a)
{
    const KsPoint k = ks_point(p, a);
    const double lu = k.lx * u.x + k.ly * u.y + k.lz * u.z, L = lu + u.w, L2 = L * L;
    const double xu = p.x * u.x + p.y * u.y + p.z * u.z, N = u.x * u.x + u.y * u.y + u.z * u.z - lu * lu;
    const double at = a * k.ta, du = -k.ka * xu - at * u.z;
    const double B = L * du + k.a2 * N - M * k.al * L2 * (k.a2 - k.b2);
    const double c = 2.0 * k.al * k.be * L, h = 0.5 * L2, hk = h * k.ka;
    return {c * (k.ly * u.z - k.lz * u.y) - B * k.lx - hk * p.x, c * (k.lz * u.x - k.lx * u.z) - B * k.ly - hk * p.y,
            c * (k.lx * u.y - k.ly * u.x) - B * k.lz - hk * p.z - h * at, B};
}

PRR_DEV void geod_vjp(const V4<double> &p, const V4<double> &u, double M, double a, const double w[4], double gx[3],
                      double gu[4], double &gM, double &ga)
{
    const KsPoint k = ks_point(p, a);
    const double X = p.x, Y = p.y, Z = p.z, ux = u.x, uy = u.y, uz = u.z, wx = w[0], wy = w[1], wz = w[2];
    const double al = k.al, be = k.be, ab = al * be, g = k.a2 - k.b2, at = a * k.ta;
    const double lu = k.lx * ux + k.ly * uy + k.lz * uz, L = lu + u.w, L2 = L * L, h = 0.5 * L2;
    const double om = k.lx * wx + k.ly * wy + k.lz * wz - w[3];
    const double cx = uy * wz - uz * wy, cy = uz * wx - ux * wz, cz = ux * wy - uy * wx;  // u x w
    const double T = k.lx * cx + k.ly * cy + k.lz * cz;
    const double xu = X * ux + Y * uy + Z * uz, xw = X * wx + Y * wy + Z * wz;
    const double N = ux * ux + uy * uy + uz * uz - lu * lu;
    const double du = -k.ka * xu - at * uz, dw = -k.ka * xw - at * wz;  // u.grad alpha, w.grad alpha
    const double ML2 = M * L2, aML2 = al * ML2;
    const double B = L * du + k.a2 * N - aML2 * g;
    const double LT = L * T, ab2 = ab + ab, kT = ab2 * L;
    // Psi and its M derivative: w.G = 2M Psi, with one more M in B
    const double Psi = h * dw + ab2 * LT - om * B;
    gM = 2.0 * (Psi + om * aML2 * g);
    // partial derivatives of Psi
    const double P_du = -om * L, P_N = -om * k.a2;
    const double P_L = ab2 * T + L * dw - om * (du - 2.0 * M * al * L * g);
    const double P_lu = P_L - 2.0 * P_N * lu;  // dPsi/dT = kT, dPsi/d(l.w) = -B, dPsi/d(w.grad alpha) = h
    const double P_ka = -(P_du * xu + h * xw), qz = P_du * uz + h * wz, P_ta = -a * qz;
    const double g3 = 3.0 * g, ab6 = 6.0 * ab;
    const double P_al = 2.0 * be * LT - om * (2.0 * al * N - ML2 * (g + 2.0 * k.a2)) + g3 * P_ka + ab6 * P_ta;
    const double P_be = 2.0 * al * LT - 2.0 * om * be * aML2 - ab6 * P_ka + g3 * P_ta;
    // through l: v = dPsi/dl, then J v = alpha (v - l (l.v)) - beta (v x l)
    const double vx = P_lu * ux - B * wx + kT * cx, vy = P_lu * uy - B * wy + kT * cy, vz = P_lu * uz - B * wz + kT * cz;
    const double lv = k.lx * vx + k.ly * vy + k.lz * vz;
    const double mx = -k.ka * P_al - k.ta * P_be, kd = k.ka * P_du, kh = k.ka * h;
    gx[0] = al * (vx - k.lx * lv) - be * (vy * k.lz - vz * k.ly) + mx * X - kd * ux - kh * wx;
    gx[1] = al * (vy - k.ly * lv) - be * (vz * k.lx - vx * k.lz) + mx * Y - kd * uy - kh * wy;
    gx[2] = al * (vz - k.lz * lv) - be * (vx * k.ly - vy * k.lx) + mx * Z - kd * uz - kh * wz + a * (k.ka * P_be - k.ta * P_al);
    const double N2 = P_N + P_N;
    gu[0] = P_lu * k.lx + N2 * ux + kT * (wy * k.lz - wz * k.ly) - kd * X;
    gu[1] = P_lu * k.ly + N2 * uy + kT * (wz * k.lx - wx * k.lz) - kd * Y;
    gu[2] = P_lu * k.lz + N2 * uz + kT * (wx * k.ly - wy * k.lx) - kd * Z - at * P_du;
    gu[3] = P_L;
    // a at fixed x: R_a = i (z + i a) / R, and l through r and explicitly
    const double ra = Z * be - a * al, k2 = 2.0 * (k.r * ra + a);
    const double la = (vx * (ra * X + Y - k.lx * k2) + vy * (ra * Y - X - k.ly * k2)) * k.iq - vz * k.lz * ra * k.ir;
    ga = P_al * (k.ka * a - k.ta * Z) + P_be * (k.ka * Z + at) + la - k.ta * qz;
}

}  // namespace prr
