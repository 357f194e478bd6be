// k_reference.cu - REFERENCE-mode tracing kernel: one thread per ray, with
// ray placement, initRays, trace_RKF/trace_Euler and rayToRGB fused (the
// reference runs them as separate launches, prr.cpp:258-323; fusing them
// changes no arithmetic).  Built with -fmad=false.
//
// Bound: FP32 issue (a quarter of it in the two powf of each Schwarzschild
// geodesic) and, on small frames, the longest ray.  The sixth stage and the
// error are evaluated only where they can decide something, and the sphere
// test only near a sphere (ref_stepper.cuh): 1920x1080x4 Kerr frame at eps
// 1e-3 813 -> 628 ms, 320x180x4 64 -> 51 ms, 320x180 Schwarzschild 13.8 ->
// 11.3 ms, the same bits.  The Kerr geodesic has a kernel of its own: with both
// geodesics at each of the six stages these frames took 628, 51 and 11.3
// ms, with one they take 580, 43 and 10.7.
#include "kernels.cuh"
#include "ref_stepper.cuh"

namespace prr {

__device__ __forceinline__ void warp_add(unsigned long long *p, unsigned long long v)
{
    unsigned mask = __activemask();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o);
    if ((threadIdx.x & 31) == (__ffs(mask) - 1)) atomicAdd(p, v);
}

template <bool KERR>
__global__ void __launch_bounds__(128) k_ref_trace(const FrameParams *__restrict__ fps, int frame, long long nrays,
                                                   float *__restrict__ state, float *__restrict__ rgb,
                                                   unsigned long long *__restrict__ counters)
{
    long long rid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (rid >= nrays) return;
    const FrameParams &fp = fps[frame];
    int S = fp.samples;
    long long pix = rid / S;
    int s = (int)(rid - pix * S);
    int x = (int)(pix % fp.width), y = (int)(pix / fp.width);
    RefRay R;
    const BuiltinHooks<KERR> hk{fp};
    ref_init_h(fp, hk, x, y, s, R);
    if (fp.solver == PRR_SOLVER_EULER) ref_euler_h(fp, hk, R);
    else ref_rkf_h(fp, hk, R);
    V3<float> c = ray_colour<float>(fp, R.result, R.r, R.u);
    if (state) {
        float *o = state + 12 * rid;
        o[0] = R.uvx; o[1] = R.uvy; o[2] = (float)R.result;
        o[3] = R.r.x; o[4] = R.r.y; o[5] = R.r.z; o[6] = R.r.w;
        o[7] = R.u.x; o[8] = R.u.y; o[9] = R.u.z; o[10] = R.u.w;
        o[11] = (float)R.accepted;
    }
    if (rgb) {
        rgb[3 * rid] = c.x; rgb[3 * rid + 1] = c.y; rgb[3 * rid + 2] = c.z;
    }
    if (counters) {
        warp_add(&counters[C_RAYS], 1ull);
        warp_add(&counters[C_ATTEMPTS], (unsigned long long)R.attempts);
        warp_add(&counters[C_ACCEPTED], (unsigned long long)R.accepted);
        float r = metric_radius<float>(fp, R.r.x, R.r.y, R.r.z);
        int cls = R.result == PRR_RESULT_SUCCESS ? (r >= fp.rout ? C_ESCAPED : C_CAPTURED)
                : R.result == PRR_RESULT_INTERSECTION ? C_INTERSECTION
                : R.result == PRR_RESULT_INFINITE_GEO ? C_INFINITE : C_MATH_ERROR;
        atomicAdd(&counters[cls], 1ull);
    }
}

cudaError_t launch_ref_trace(const FrameParams &fp, const FrameParams *d_fp, int frame, long long nrays, float *state, float *rgb,
                             unsigned long long *counters, cudaStream_t st)
{
    if (nrays <= 0) return cudaSuccess;
    // a warp leaves when its longest ray does: one-warp CTAs free their slots at once, which a frame of about a wave
    // likes (320x180 Schwarzschild 10.7 ms against 11.3 with four warps, 640x360 Kerr 43.8 and 44.4), and a large one not
    // (1920x1080x4: 582 and 580), nor one whose eps is so tight that rays take up to 10^6 attempts (96x54 at eps 1e-6: 4.78 s
    // against 4.56)
    const int block = ref_bounded(fp) && nrays <= (1 << 19) ? 32 : 128;
    long long grid = (nrays + block - 1) / block;
    auto k = fp.metric == PRR_METRIC_KERR ? k_ref_trace<true> : k_ref_trace<false>;
    k<<<(unsigned)grid, block, 0, st>>>(d_fp, frame, nrays, state, rgb, counters);
    return cudaGetLastError();
}

}  // namespace prr
