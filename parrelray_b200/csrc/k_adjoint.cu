// k_adjoint.cu - discrete adjoint of the PHYSICAL-mode RKF45 render:
// d(loss)/d(spin a, mass M, camera inclination i, camera distance r, orbital
// phase of one sphere) given dL/d(image).
//
// Per ray, with the accepted step sizes and every discrete event
// (accept/reject, intersection mode, termination, which sphere is hit)
// frozen at the forward run.  The forward steps run in the frame's precision
// (TF = float: the FP32 PHYSICAL stepper with Kahan-compensated updates;
// TF = double: FP64); the adjoint and the gradient reduction are FP64:
//   1. forward: the PHYSICAL stepper runs the ray and stores, in HBM, the state
//      and the step length of every accepted step (a window of `cap` steps per
//      thread), and its full state at the start of each window (checkpoints);
//   2. colour adjoint: dL/dc of the ray's sample through the SSAA combine,
//      then lambda_N = dL/dc . dc/dy_N (+ the sphere-phase term) with c the
//      bilinear sky or the sphere texture at the hit point;
//   3. reverse: lambda is pulled back through each step, last first, from
//      the stored states.  Rays longer than a window recompute the earlier ones
//      from their checkpoints (bit-identical: same stepper).  Each step of
//      x' = u, u' = G(x, u) is taken in the stepper's form (only the velocity
//      increments ku_i = h G(z_i) are kept: the stage points z_i are rebuilt from
//      them, and their adjoints carry the position coupling); the products
//      lambda^T dG/dz come from the geodesic's hand-written reverse sweep
//      (geod_vjp.cuh);
//   4. lambda_0 is pulled back through the initial data (camera position,
//      ray direction, null u^t), also by dual numbers.
// Gradients are accumulated per thread and reduced in FP64.
//
// Bound: FP64 latency at 8 (FP64 steps) or 12 warps per SM.  On 512x512 with
// FP32 steps the sixth stage's zero products, two recompute passes per step
// and a fixed assignment of rays to threads cost 117 ms, without them 59 ms,
// and with the closed forms of geod_vjp.cuh 37 ms (256x256 with FP64 steps:
// 64.7, 41.5, 31.5 and, with adj_attempt's rule, 27.4 ms); windows of 4096
// steps, which hold the longest rays (kernels.cuh), took 3 and 6 ms more off.
// The states are 36 bytes per FP32 step, 11 GB written and read per 512x512
// gradient: 3.4 ms of HBM time spread under the arithmetic.
#include <cub/device/device_radix_sort.cuh>

#include "dual.cuh"
#include "geod_vjp.cuh"
#include "kernels.cuh"
#include "phys_stepper.cuh"

namespace prr {

using DC = Dual<13>;  // initial data / colour: 8 state components + 5 parameters
enum { P_SPIN = 0, P_MASS = 1, P_INCL = 2, P_CAMR = 3, P_PHASE = 4 };

// Sphere::getColor at p + v d for a T-valued centre (derivative-carrying
// version of sphere_colour; same arithmetic in FP64).
template <class T>
__device__ V3<T> sphere_colour_ad(const DevSphere &S, T cx, T cy, T cz, T px, T py, T pz, T vx, T vy, T vz, T d)
{
    T ix = (px + vx * d) - cx, iy = (py + vy * d) - cy, iz = (pz + vz * d) - cz, rad = (T)(double)S.r;
    T theta = acos(iz / rad);
    T phi = atan2(iy, ix) + (T)PI_SPHERE;
    T uu = phi / (T)(2.0 * PI_SPHERE), vv = theta / (T)PI_SPHERE;
    const T uvmax = (T)(double)0.999999999f;
    uu = fmin(fmax(uu, (T)0.0), uvmax);
    vv = fmin(fmax(vv, (T)0.0), uvmax);
    V3<T> col = {(T)0.5, (T)0.5, (T)0.5};
    if (S.tex.p) col = tex_bilinear<T>(S.tex, uu, vv);
    T shade = fmax((T)0.0, fmin((T)0.5 + (T)0.5 * iz / rad, (T)1.0));
    return {col.x * shade, col.y * shade, col.z * shade};
}

// Orbit camera and scene parameters of the frame, with the parameter
// derivatives seeded (tangent 8 + parameter index).
struct AdjParams {
    double spin, mass, incl, cam_r, phase, sph_R, sph_z;
    int sphere;  // index of the sphere whose phase is differentiated (-1: none)
};

__device__ void initial_state(const FrameParams &fp, const AdjParams &ap, float uvx, float uvy, double y[8], double dy[8][5])
{
    DC a = DC::var(ap.spin, 8 + P_SPIN), M = DC::var(ap.mass, 8 + P_MASS);
    DC inc = DC::var(ap.incl, 8 + P_INCL), r = DC::var(ap.cam_r, 8 + P_CAMR);
    if (fp.metric != PRR_METRIC_KERR) a = DC(0.0);
    if (fp.metric == PRR_METRIC_FLAT) M = DC(0.0);
    DC px = r * sin(inc), py = DC(0.0), pz = r * cos(inc);
    // Camera::rayDir_Spherical with a = pi, b = i - pi/2
    const double PI = 3.14159265358979323846;
    DC beta = inc - DC(0.5 * PI);
    double nu = (0.5 - (double)uvy) * (double)fp.vfov;
    double mu = (0.5 - (double)uvx) * (double)fp.width / (double)fp.height * (double)fp.vfov;
    DC cb = cos(beta + DC(nu));
    DC dx = cb * ::cos(PI + mu), dyv = cb * ::sin(PI + mu), dz = sin(beta + DC(nu));
    DC k = DC(1.0) / sqrt(dx * dx + dyv * dyv + dz * dz);
    dx = dx * k; dyv = dyv * k; dz = dz * k;
    DC g[16];
    metric_ks<DC>(px, py, pz, M, a, g);
    DC A = g[15];
    DC Bq = DC(2.0) * (g[12] * dx + g[13] * dyv + g[14] * dz);
    DC Cq = g[0] * dx * dx + g[5] * dyv * dyv + g[10] * dz * dz + DC(2.0) * (g[1] * dx * dyv + g[2] * dx * dz + g[6] * dyv * dz);
    DC rt = sqrt(Bq * Bq - DC(4.0) * A * Cq);
    DC u0 = fmax((-Bq + rt) / (DC(2.0) * A), (-Bq - rt) / (DC(2.0) * A));
    if (u0 < 0.0) u0 = DC(1.0);
    const DC s[8] = {px, py, pz, DC(0.0), dx, dyv, dz, u0};
    for (int c = 0; c < 8; c++) {
        y[c] = s[c].v;
        for (int p = 0; p < 5; p++) dy[c][p] = s[c].d[8 + p];
    }
}

// Fehlberg coefficients for runtime stage indices: A (stage weights), B = A*A
// (the position stages, phys_stepper.cuh) and c = A*1.
__constant__ double c_A[6][5] = {{0, 0, 0, 0, 0},
                                 {Fehlberg::A21, 0, 0, 0, 0},
                                 {Fehlberg::A31, Fehlberg::A32, 0, 0, 0},
                                 {Fehlberg::A41, Fehlberg::A42, Fehlberg::A43, 0, 0},
                                 {Fehlberg::A51, Fehlberg::A52, Fehlberg::A53, Fehlberg::A54, 0},
                                 {Fehlberg::A61, Fehlberg::A62, Fehlberg::A63, Fehlberg::A64, Fehlberg::A65}};
__constant__ double c_B[6][5] = {{0, 0, 0, 0, 0},
                                 {0, 0, 0, 0, 0},
                                 {Fehlberg::B31, 0, 0, 0, 0},
                                 {Fehlberg::B41, Fehlberg::B42, 0, 0, 0},
                                 {Fehlberg::B51, Fehlberg::B52, Fehlberg::B53, 0, 0},
                                 {Fehlberg::B61, Fehlberg::B62, Fehlberg::B63, Fehlberg::B64, 0}};
__constant__ double c_c[6] = {0.0, Fehlberg::c2, Fehlberg::c3, Fehlberg::c4, Fehlberg::c5, Fehlberg::c6};
__constant__ double c_K4[6] = {Fehlberg::K41, Fehlberg::K42, Fehlberg::K43, Fehlberg::K44, Fehlberg::K45, Fehlberg::K46};
__constant__ double c_beta[6] = {Fehlberg::b1, Fehlberg::b2, Fehlberg::b3, Fehlberg::b4, Fehlberg::b5, 0.0};

// Stage point i of the Fehlberg step from y = (x, u), h and the velocity
// increments ku_0..ku_{i-1} (x' = u is linear in the stages: phys_stepper.cuh):
//   z_i^u = u + sum_m A_im ku_m,  z_i^x = x + h (c_i u + sum_m B_im ku_m).
__device__ __forceinline__ void stage_point(const double y[8], double h, const double ku[4][4], int i, V4<double> &zx,
                                            V4<double> &zu)
{
    double sx[4], su[4];
#pragma unroll
    for (int c = 0; c < 4; c++) { su[c] = y[4 + c]; sx[c] = c_c[i] * y[4 + c]; }
    for (int m = 0; m < i; m++)
#pragma unroll
        for (int c = 0; c < 4; c++) { su[c] += c_A[i][m] * ku[m][c]; sx[c] += c_B[i][m] * ku[m][c]; }
    zx = {y[0] + h * sx[0], y[1] + h * sx[1], y[2] + h * sx[2], y[3] + h * sx[3]};
    zu = {su[0], su[1], su[2], su[3]};
}

// lambda <- lambda . dPhi/dy at (y, h), Phi the 4th-order Fehlberg step
//   u+ = u + sum_m K4_m ku_m,  x+ = x + h (u + sum_m beta_m ku_m);
// th[0..1] += lambda . dPhi/d(spin, mass).  Only the first four velocity
// increments ku (16 doubles) and the adjoints of the first five (20 doubles)
// are kept; the stage points are rebuilt from them.
__device__ void step_vjp(const Hot<double> &q, const double y[8], double h, double lam[8], double th[2])
{
    if (q.metric == PRR_METRIC_FLAT) {  // G = 0: x+ = x + h u
#pragma unroll
        for (int c = 0; c < 4; c++) lam[4 + c] += h * lam[c];
        return;
    }
    // The 4th-order step has no weight on the sixth stage (K46 = 0), so its adjoint is zero and the fifth
    // increment, which only the sixth stage point uses, is not needed: four forward stages, five reverse ones.
    const double hm = 2.0 * q.M * h;  // geod_unit and geod_vjp leave the 2M to the step length
    double ku[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        V4<double> zx, zu;
        stage_point(y, h, ku, i, zx, zu);
        const V4<double> g = geod_unit(zx, zu, q.M, q.a);
        ku[i][0] = hm * g.x; ku[i][1] = hm * g.y; ku[i][2] = hm * g.z; ku[i][3] = hm * g.w;
    }
    // adjoints of the outputs: of ku_m, and of (x, u) through the direct terms
    double kb[5][4], ox[4], ou[4];
#pragma unroll
    for (int c = 0; c < 4; c++) {
        // (lam[3], of the coordinate time, is zero throughout: no colour and no acceleration depends on it)
        ox[c] = c < 3 ? lam[c] : 0.0;
        ou[c] = lam[4 + c] + h * ox[c];
#pragma unroll
        for (int m = 0; m < 5; m++) kb[m][c] = c_K4[m] * lam[4 + c] + (h * c_beta[m]) * ox[c];
    }
#pragma unroll 1
    for (int i = 4; i >= 0; i--) {
        V4<double> zx, zu;
        stage_point(y, h, ku, i, zx, zu);
        double gx[3], gu[4], gM, ga;
        const double wv[4] = {kb[i][0], kb[i][1], kb[i][2], kb[i][3]};
        geod_vjp(zx, zu, q.M, q.a, wv, gx, gu, gM, ga);
        th[0] += hm * ga;
        th[1] += h * gM;
        // adjoints of the stage point (nothing depends on the coordinate time)
        double zbx[3], zbu[4];
#pragma unroll
        for (int c = 0; c < 4; c++) {
            zbu[c] = hm * gu[c];
            ou[c] += zbu[c];
        }
#pragma unroll
        for (int c = 0; c < 3; c++) {
            zbx[c] = hm * gx[c];
            ox[c] += zbx[c];
            ou[c] += h * c_c[i] * zbx[c];
        }
        for (int m = 0; m < i; m++) {
            const double A = c_A[i][m], hB = h * c_B[i][m];
#pragma unroll
            for (int c = 0; c < 4; c++) kb[m][c] += A * zbu[c];
#pragma unroll
            for (int c = 0; c < 3; c++) kb[m][c] += hB * zbx[c];
        }
    }
#pragma unroll
    for (int c = 0; c < 4; c++) { lam[c] = ox[c]; lam[4 + c] = ou[c]; }
}

struct AdjointArgs {
    const FrameParams *frame;  // device, one frame
    AdjParams ap;
    const float *dL_dimage;    // W*H*3 (device)
    const float *image;        // forward combined image W*H*3 (device)
    void *ckpt;                // per thread: max_ckpt checkpoints (PhysRay<TF>), one per window
    int max_ckpt;
    void *states;              // cap x ADJ_STATE values (TF) per thread, thread index fastest
    int cap;                   // accepted steps per window
    double *grad;              // 5 doubles, accumulated
    unsigned long long *counters;
    long long nrays;
    const unsigned *order;     // ray visit order (null: 0, 1, 2, ...)
};

constexpr int ADJ_STATE = 9;  // values stored per accepted step: the state before it (x, u) and its length h

// Resident CTAs of 128 threads per SM the kernel is built for (caps the
// registers): FP32 steps 3 (168 registers: 36.8 ms on 512x512 against 38.9
// with 255), FP64 steps 2 (255 registers: 31.4 ms on 256x256 against 38.8
// with 168).
template <class TF> constexpr int adj_minb() { return sizeof(TF) == 4 ? 3 : 2; }

template <class TF> __device__ __forceinline__ void state8(const PhysRay<TF> &R, double y[8])
{
    y[0] = (double)R.x.x; y[1] = (double)R.x.y; y[2] = (double)R.x.z; y[3] = (double)R.x.w;
    y[4] = (double)R.u.x; y[5] = (double)R.u.y; y[6] = (double)R.u.z; y[7] = (double)R.u.w;
}

// One RKF45 attempt of the adjoint's own forward steps.  The forward pass and
// the recomputed windows go through this one out-of-line copy, so a recomputed
// window repeats the forward steps bit for bit: inlined copies of the same
// source may contract multiply-adds differently, and a recomputed step
// sequence that drifts from the forward one would pull lambda back through
// steps that were never taken.
// FP64 steps evaluate the sixth stage and the error only where they can
// decide something (cruise_radius, r2 its square for R^2; nor in intersection
// mode, which accepts hmin steps whatever the error until its 10000 attempts
// are used up), for a warp when one of its lanes needs them: 256x256 gradient
// 31.5 -> 27.4 ms.  FP32 steps run beside the FP64 sweeps of other warps and
// gain nothing from it (512x512: 36.9 against 37.4 ms, with more spills).
template <class TF>
__device__ __noinline__ int adj_attempt(const FrameParams &fp, const Hot<TF> &q, PhysRay<TF> &R, float r2, int &result,
                                        V3<float> &col, int &hit)
{
    bool full = true;
    if constexpr (sizeof(TF) == 8) {
        const bool quiet = (R.intersect && R.i < 10000) ||
                           (R.h == q.hmax && (float)(R.x.x * R.x.x + R.x.y * R.x.y + R.x.z * R.x.z) >= r2);
        full = __any_sync(__activemask(), !quiet);
    }
    return phys_attempt<TF, 0>(fp, q, R, result, col, (TF)-1, &hit, nullptr, full);
}

// cruise_radius^2 + a^2 (bounds the Kerr-Schild r by the Euclidean R) for the initial state y, infinite when y is not null.
__device__ float adj_cruise_r2(const FrameParams &fp, double M, double a, const double y[8], float noise)
{
    double g[16], p[4], n = 0.0, t = 0.0;
    metric_ks<double>(y[0], y[1], y[2], M, a, g);
    for (int m = 0; m < 4; m++) {
        p[m] = g[4 * m] * y[4] + g[4 * m + 1] * y[5] + g[4 * m + 2] * y[6] + g[4 * m + 3] * y[7];
        n += p[m] * y[4 + m];
        t += fabs(p[m] * y[4 + m]);
    }
    if (!(fabs(n) <= 1e-3 * t)) return INFINITY;
    const float r = cruise_radius(fp, fabsf((float)p[3]), (float)M, noise);
    return 1.0001f * (r * r + (float)(a * a));
}

// lambda_N = gc . dc/dy_N of a ray that shows the sky (escaped) or sphere `hit`, and the direct phase term.
template <class TF>
__device__ __noinline__ void colour_adjoint(const FrameParams &fp, const AdjParams &ap, const PhysRay<TF> &R, bool escaped, int hit,
                                            const double gc[3], double lam[8], double &phase_c)
{
    DC st[8];
    double yN[8];
    state8(R, yN);
    for (int c = 0; c < 8; c++) st[c] = DC::var(yN[c], c);
    V3<DC> cd;
    if (escaped) {
        cd = background_bilinear<DC>(fp.bg, st[4], st[5], st[6]);
        if (!fp.bg.p || fp.bg_filter != PRR_BG_BILINEAR) cd = {DC(0.0), DC(0.0), DC(0.0)};  // RMS2X2 is piecewise constant
    } else {
        const DevSphere &Sp = fp.sph[hit];
        DC cx = DC((double)Sp.cx), cy = DC((double)Sp.cy), cz = DC((double)Sp.cz);
        if (hit == ap.sphere) {
            DC ph = DC::var(ap.phase, 8 + P_PHASE);
            cx = DC(ap.sph_R) * cos(ph); cy = DC(ap.sph_R) * sin(ph); cz = DC(ap.sph_z);
        }
        DC k = DC(1.0) / sqrt(st[4] * st[4] + st[5] * st[5] + st[6] * st[6]);
        DC vx = st[4] * k, vy = st[5] * k, vz = st[6] * k;
        DC v2 = vx * vx + vy * vy + vz * vz;
        DC dx = st[0] - cx, dy = st[1] - cy, dz = st[2] - cz;
        DC dvp = vx * dx + vy * dy + vz * dz;
        DC disc = dvp * dvp - v2 * ((dx * dx + dy * dy + dz * dz) - DC((double)Sp.r * (double)Sp.r));
        DC d = (DC(-2.0) * dvp - sqrt(disc)) / v2;
        cd = sphere_colour_ad<DC>(Sp, cx, cy, cz, st[0], st[1], st[2], vx, vy, vz, d);
    }
    const DC *cc3 = &cd.x;
    for (int c = 0; c < 3; c++) {
        for (int j = 0; j < 8; j++) lam[j] += gc[c] * cc3[c].d[j];
        phase_c += gc[c] * cc3[c].d[8 + P_PHASE];
    }
}

template <class TF> __global__ void __launch_bounds__(128, adj_minb<TF>()) k_adjoint(AdjointArgs A)
{
    const FrameParams &fp = *A.frame;
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long nth = (long long)gridDim.x * blockDim.x;
    PhysRay<TF> *ck = (PhysRay<TF> *)A.ckpt + tid * A.max_ckpt;
    Hot<TF> qf = make_hot<TF>(fp);
    qf.a = fp.metric == PRR_METRIC_KERR ? (TF)A.ap.spin : (TF)0;
    qf.M = fp.metric == PRR_METRIC_FLAT ? (TF)0 : (TF)A.ap.mass;
    Hot<double> q = make_hot<double>(fp);  // the adjoint's (FP64) copy
    q.a = fp.metric == PRR_METRIC_KERR ? A.ap.spin : 0.0;
    q.M = fp.metric == PRR_METRIC_FLAT ? 0.0 : A.ap.mass;
    double gacc[5] = {0, 0, 0, 0, 0};
    unsigned long long n_bad = 0, n_steps = 0;
    const int S = fp.samples;
    // slot-major, thread index fastest: a warp's lanes, whose rays have similar lengths, read and write lines
    TF *const mine = (TF *)A.states + tid;
    auto slot = [&](int n, int c) -> TF & { return mine[((long long)(n % A.cap) * ADJ_STATE + c) * nth]; };
    auto keep = [&](int n, const TF y[8], TF h) {
#pragma unroll
        for (int c = 0; c < 8; c++) slot(n, c) = y[c];
        slot(n, 8) = h;
    };
    // A warp takes the next 32 rays of the order (longest first) when its last 32 are done.  Its lanes meet again after
    // the forward steps and walk the reverse sweep by a common step index (idle where their ray is shorter): left to
    // themselves they ran it in groups, at 21 of 32 lanes.
    while (true) {
        long long k = 0;
        if (lane == 0) k = (long long)atomicAdd(&A.counters[C_WORK], 32ull);
        k = __shfl_sync(FULL, k, 0);
        if (k >= A.nrays) break;
        k += lane;
        int N = 0;  // steps to pull lambda back through; 0: no gradient (black, or no weight)
        double dy0[8][5];
        double lam[8] = {0, 0, 0, 0, 0, 0, 0, 0}, th[2] = {0, 0}, phase_c = 0.0;
        float cr2 = INFINITY;
        if (k < A.nrays) {
            const long long rid = A.order ? (long long)A.order[k] : k;
            long long pix = rid / S;
            int s = (int)(rid - pix * S);
            int px = (int)(pix % fp.width), py = (int)(pix / fp.width);
            // dL/dc through the SSAA combine (kernels/ssaa.cuh:116-130)
            float uvx, uvy;
            ray_uv(fp, px, py, s, uvx, uvy);
            double y0[8];
            initial_state(fp, A.ap, uvx, uvy, y0, dy0);
            PhysRay<TF> R;
            R.x = {(TF)y0[0], (TF)y0[1], (TF)y0[2], (TF)y0[3]};
            R.u = {(TF)y0[4], (TF)y0[5], (TF)y0[6], (TF)y0[7]};
            R.cx = {0, 0, 0, 0}; R.cu = {0, 0, 0, 0};
            R.h = (TF)fp.h; R.trace_h = (TF)fp.h; R.l = 0; R.i = 0; R.accepted = 0; R.intersect = 0;
            if constexpr (sizeof(TF) == 8) cr2 = adj_cruise_r2(fp, q.M, q.a, y0, cruise_noise<TF>());
            ck[0] = R;
            int result = 0, hit = -1;
            V3<float> col;
            bool ok = true;
            while (true) {
                const int before = R.accepted;
                const TF yb[8] = {R.x.x, R.x.y, R.x.z, R.x.w, R.u.x, R.u.y, R.u.z, R.u.w};
                const TF hb = R.h;
                const int st = adj_attempt<TF>(fp, qf, R, cr2, result, col, hit);
                if (R.accepted > before) {
                    keep(before, yb, hb);
                    if (st == STEP_CONTINUE && R.accepted % A.cap == 0) {
                        const int w = R.accepted / A.cap;
                        if (w >= A.max_ckpt) { ok = false; break; }
                        ck[w] = R;
                    }
                }
                if (st != STEP_CONTINUE) break;
            }
            if (ok) n_steps += (unsigned long long)R.accepted;
            else n_bad++;
            const bool escaped = result == PRR_RESULT_SUCCESS && metric_radius<TF>(fp, R.x.x, R.x.y, R.x.z) >= (TF)fp.rout;
            if (ok && (escaped || result == PRR_RESULT_INTERSECTION)) {
                // dL/dc for this sample
                const float *gI = A.dL_dimage + 3 * pix;
                const float *I = A.image + 3 * pix;
                double gc[3];
                const float cc[3] = {col.x, col.y, col.z};
                bool any = false;
                for (int c = 0; c < 3; c++) {
                    double d;
                    if (S == 1) d = (cc[c] > 0.0f && cc[c] < 1.0f) ? 1.0 : 0.0;
                    else d = (cc[c] * cc[c] > 0.0f && cc[c] * cc[c] < 1.0f && I[c] > 0.0f) ? (double)cc[c] / ((double)S * I[c]) : 0.0;
                    gc[c] = (double)gI[c] * d;
                    any |= gc[c] != 0.0;
                }
                if (any) {
                    N = R.accepted;
                    colour_adjoint<TF>(fp, A.ap, R, escaped, hit, gc, lam, phase_c);
                }
            }
        }
        __syncwarp(FULL);
        // reverse sweep, window by window; the last window's states are in
        // place.  A recomputation that does not reach the steps the forward
        // pass took (it cannot, as both run the same code, but it is checked
        // rather than trusted) drops the ray: its states would be missing.
        bool live = N > 0;
        const int most = __reduce_max_sync(FULL, N);
        for (int w = (most - 1) / A.cap; w >= 0 && most > 0; w--) {
            const int lo = w * A.cap, hi = min(N, lo + A.cap);
            if (live && N > lo + A.cap) {
                int r2 = 0, h2 = -1;
                V3<float> c2;
                PhysRay<TF> Rs = ck[w];
                while (Rs.accepted < hi) {
                    const int before = Rs.accepted;
                    const TF yb[8] = {Rs.x.x, Rs.x.y, Rs.x.z, Rs.x.w, Rs.u.x, Rs.u.y, Rs.u.z, Rs.u.w};
                    const TF hb = Rs.h;
                    const int st = adj_attempt<TF>(fp, qf, Rs, cr2, r2, c2, h2);
                    if (Rs.accepted > before) keep(before, yb, hb);
                    if (st != STEP_CONTINUE) break;
                }
                if (Rs.accepted != hi) live = false;
            }
            __syncwarp(FULL);
            const int top = min(most, lo + A.cap) - 1, from = live ? hi : 0;  // this lane's steps: lo <= n < from
            TF next[ADJ_STATE];
            if (top < from) {
#pragma unroll
                for (int c = 0; c < ADJ_STATE; c++) next[c] = slot(top, c);
            }
#pragma unroll 1
            for (int n = top; n >= lo; n--) {
                double y[8];
#pragma unroll
                for (int c = 0; c < 8; c++) y[c] = (double)next[c];
                const double h = (double)next[8];
                if (n > lo && n - 1 < from) {  // the next state's loads fly during this step's products
#pragma unroll
                    for (int c = 0; c < ADJ_STATE; c++) next[c] = slot(n - 1, c);
                }
                if (n < from) step_vjp(q, y, h, lam, th);
                __syncwarp(FULL);
            }
        }
        if (N > 0 && !live) n_bad++;
        if (live) {
            gacc[P_PHASE] += phase_c;
            gacc[P_SPIN] += th[0];
            gacc[P_MASS] += th[1];
            for (int c = 0; c < 8; c++)
                for (int p = 0; p < 5; p++) gacc[p] += lam[c] * dy0[c][p];
        }
    }
    for (int p = 0; p < 5; p++) {
        double v = gacc[p];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0 && v != 0.0) atomicAdd(&A.grad[p], v);
    }
    if (n_bad) atomicAdd(&A.counters[C_MATH_ERROR], n_bad);
    atomicAdd(&A.counters[C_ACCEPTED], n_steps);
}

cudaError_t launch_adjoint(const FrameParams *d_fp, const AdjointParamsHost &p, const float *dL, const float *image,
                           void *ckpt, int max_ckpt, void *states, int cap, int threads_total, double *grad,
                           unsigned long long *counters, long long nrays, const unsigned *order, int precision, cudaStream_t st)
{
    AdjointArgs A;
    A.frame = d_fp;
    A.ap = {p.spin, p.mass, p.incl, p.cam_r, p.phase, p.sph_R, p.sph_z, p.sphere};
    A.dL_dimage = dL;
    A.image = image;
    A.ckpt = ckpt;
    A.max_ckpt = max_ckpt;
    A.states = states;
    A.cap = cap;
    A.grad = grad;
    A.counters = counters;
    A.nrays = nrays;
    A.order = order;
    if (precision == PRR_PREC_FP32) k_adjoint<float><<<threads_total / 128, 128, 0, st>>>(A);
    else k_adjoint<double><<<threads_total / 128, 128, 0, st>>>(A);
    return cudaGetLastError();
}

__global__ void k_iota(unsigned *v, long long n)
{
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) v[i] = (unsigned)i;
}

// scratch layout: [iota values | sorted keys | cub temporary storage]
size_t adjoint_order_bytes(long long nrays)
{
    size_t temp = 0;
    cub::DeviceRadixSort::SortPairsDescending(nullptr, temp, (const int *)nullptr, (int *)nullptr,
                                              (const unsigned *)nullptr, (unsigned *)nullptr, (int)nrays);
    const size_t n4 = ((size_t)nrays * 4 + 255) / 256 * 256;
    return 2 * n4 + temp + 256;
}

cudaError_t launch_adjoint_order(const int *steps, long long nrays, unsigned *order, void *scratch, cudaStream_t st)
{
    if (nrays <= 0) return cudaSuccess;
    const size_t n4 = ((size_t)nrays * 4 + 255) / 256 * 256;
    unsigned *iota = (unsigned *)scratch;
    int *keys_out = (int *)((char *)scratch + n4);
    void *temp = (char *)scratch + 2 * n4;
    k_iota<<<(unsigned)((nrays + 255) / 256), 256, 0, st>>>(iota, nrays);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    size_t temp_bytes = 0;
    e = cub::DeviceRadixSort::SortPairsDescending(nullptr, temp_bytes, steps, keys_out, iota, order, (int)nrays);
    if (e != cudaSuccess) return e;
    return cub::DeviceRadixSort::SortPairsDescending(temp, temp_bytes, steps, keys_out, iota, order, (int)nrays, 0,
                                                     32, st);
}

size_t adjoint_checkpoint_bytes(int precision)
{
    return precision == PRR_PREC_FP32 ? sizeof(PhysRay<float>) : sizeof(PhysRay<double>);
}

size_t adjoint_state_bytes(int precision) { return ADJ_STATE * (precision == PRR_PREC_FP32 ? sizeof(float) : sizeof(double)); }

int adjoint_window(size_t budget, int threads, int max_steps, int precision)
{
    auto bytes = [&](int cap) {
        return (size_t)threads * (cap * adjoint_state_bytes(precision) + (max_steps / cap + 2) * adjoint_checkpoint_bytes(precision));
    };
    int cap = ADJ_WINDOW;
    while (cap > ADJ_WINDOW_MIN && cap / 2 >= max_steps) cap /= 2;
    while (cap > ADJ_WINDOW_MIN && bytes(cap) > budget && bytes(cap / 2) < bytes(cap)) cap /= 2;
    return cap;
}

int adjoint_blocks_per_sm(int precision)
{
    int n = 0;
    cudaError_t e = precision == PRR_PREC_FP32 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_adjoint<float>, 128, 0)
                                               : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_adjoint<double>, 128, 0);
    if (e != cudaSuccess) { cudaGetLastError(); return 1; }
    return n > 0 ? n : 1;
}

}  // namespace prr
