// sphere_path.cuh - how far a ray of k_ham's intersection mode can fly before Sphere::intersects can pass (k_ham.cu).
#pragma once
#include "prr_device.cuh"

namespace prr {

// sqrt(v) to 2^-22, for v > 0.
PRR_DEV float path_sqrt(float v) { return v * sfu_rsqrt(v); }

// Path length within which a ray of intersection mode at p, flying along the unit vector v, cannot pass
// Sphere::intersects on S with the window w (hmin): 0 or less when that cannot be said.  With rho = p - c, D = |rho|,
// b = -v.rho and disc = b^2 - (D^2 - R^2), the test's distance is d = 2b - sqrt(disc), and a hit needs 0 <= d <= sqrt(w)
// (the factor 2 lets a head-on ray fly on inside the sphere, down to D = R/2).  Along a path of curvature <= kappa, b
// falls by at most (1 + D kappa) per length and disc changes by at most 2 D^2 kappa, so over a length S
//     d >= 2 (b - S (1 + D kappa)) - sqrt(disc + 2 D^2 kappa S)
// and, where the ray has passed (d < 0), d <= 2 (b + S D kappa) - sqrt(disc - 2 D^2 kappa S).
// Curvature: over null geodesics in Kerr-Schild coordinates kappa r^2 / M is at most 4.0 at r >= 4M, 5.3 at 3.67M and
// 6.2 at 3.5M (maxima over 4 10^5 random states each).  S is at most D/5 and r/12, so D grows to at most 1.2 D and r falls to
// no less than 11/12 r: 5.3 (12/11)^2 1.2^2 < 9.1, and kappa is taken as 10 M / r^2.
// Rounding: 4e-6 D^2 under the root and 1e-5 D outside it cover the FP32 arithmetic of the test and of this bound.  The
// points of FP32 rays are rounded as well, by up to 2^-24 |p| here and at the point tested: `at` = 4e-7 max|p_i| is
// above their sum; it moves b by `at` and disc by (2 D + at) at, which counts for small spheres far from the origin.
template <class T>
PRR_DEV float sphere_path(const DevSphere &S, T px, T py, T pz, T vx, T vy, T vz, float w, float M, float r2)
{
    const float dx = (float)(px - (T)S.cx), dy = (float)(py - (T)S.cy), dz = (float)(pz - (T)S.cz);
    const float D2 = fmaxf(dx * dx + dy * dy + dz * dz, 1e-30f), D = path_sqrt(D2), sqw = path_sqrt(w);
    const float at = sizeof(T) == 4 ? 4e-7f * fmaxf(fmaxf(fabsf((float)px), fabsf((float)py)), fabsf((float)pz)) : 0.0f;
    const float away = D - 1.1f * S.r - sqw;
    if (away > 0.0f) return 0.9f * away - at;  // far from it (R^2 + w/3 bounds a hit)
    if (!(r2 >= 16.0f * M * M)) return 0.0f;
    const float b = -((float)vx * dx + (float)vy * dy + (float)vz * dz);
    const float disc = b * b - (D2 - S.r * S.r);
    const float kap = M > 0.0f ? 10.0f * M * sfu_rcp(r2) : 0.0f, grow = 2.0f * D2 * kap;
    const float err = 4e-6f * D2 + (2.0f * D + at) * at, out = 1e-5f * D + 2.0f * at, sw = 1.00001f * sqw + out;
    const float reach = M > 0.0f ? (1.0f / 12.0f) * path_sqrt(r2) : 1e30f;
    // ahead: half of the way that straight flight has left
    const float p = fmaxf(disc, 0.0f) + err;
    const float S1 = fminf(0.25f * (2.0f * b - path_sqrt(p) - sw), fminf(0.2f * D, reach));
    if (S1 > 0.0f && 2.0f * (b - S1 * (1.0f + D * kap)) - path_sqrt(p + grow * S1) > sw) return S1;
    // missing it, or passed: a fixed share of the size
    const float S2 = fminf(0.05f * D, reach);
    if (disc + grow * S2 + err < 0.0f) return S2;
    if (2.0f * (b + D * kap * S2) - path_sqrt(fmaxf(disc - grow * S2 - err, 1e-30f)) < -out) return S2;
    return 0.0f;
}

}  // namespace prr
