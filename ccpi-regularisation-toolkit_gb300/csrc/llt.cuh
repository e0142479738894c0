// LLT-ROF streaming kernels' launch plan (llt.cu, llt_pair.cu) and the
// terms that the two-voxel kernels share.
#pragma once

#include "pair.cuh"
#include "runtime.cuh"

namespace cilreg {

// dp / sqrt(s) per component
__device__ __forceinline__ float2 normalise2(float2 dp, float2 s) {
    return pair::mul2(dp, make_float2(rsqrtf(s.x), rsqrtf(s.y)));
}

// v / (|v| + 1e-12), the second difference over its magnitude (llt_term
// of llt.cu), with the IEEE quotient's value and without its division for
// almost every v: from |v| = 2^-15 on, 1e-12 is below half an ulp of |v|, so
// the rounded denominator is |v| and the quotient exactly +-1; v = +-0 gives
// itself.  Only the other values (below 2^-15, infinite, NaN) divide: a step
// forms the six terms of its pair by sign copies and, when any of them needs
// it, all six by the division (one branch).
__device__ __forceinline__ float llt_sign1(float v) { return (v == 0.0f) ? v : copysignf(1.0f, v); }
__device__ __forceinline__ float2 llt_sign2(float2 v) { return make_float2(llt_sign1(v.x), llt_sign1(v.y)); }
__device__ __forceinline__ bool llt_divides(float v) {
    const float a = fabsf(v);
    return !(a >= 0x1p-15f && a <= 3.4028234664e38f) && a != 0.0f;
}
__device__ __forceinline__ bool llt_divides2(float2 v) { return llt_divides(v.x) | llt_divides(v.y); }
__device__ __forceinline__ float2 llt_quot2(float2 v) {
    return make_float2(v.x / (fabsf(v.x) + 1.0e-12f), v.y / (fabsf(v.y) + 1.0e-12f));
}


// The terms of N second differences.  Where all of them are finite and at least
// 2^-15 (one test for all: their smallest magnitude, and the sum of the
// magnitudes, which is not finite where one of them is not), they are sign
// copies; else each is looked at by itself, as above.
template <int N>
__device__ __forceinline__ void llt_terms(const float2 (&v)[N], float2 (&t)[N]) {
    float least = fminf(fabsf(v[0].x), fabsf(v[0].y)), all = fabsf(v[0].x) + fabsf(v[0].y);
#pragma unroll
    for (int i = 1; i < N; i++) {
        least = fminf(least, fminf(fabsf(v[i].x), fabsf(v[i].y)));
        all += fabsf(v[i].x) + fabsf(v[i].y);
    }
    if (least >= 0x1p-15f && all <= 3.4028234664e38f) {
#pragma unroll
        for (int i = 0; i < N; i++) t[i] = make_float2(copysignf(1.0f, v[i].x), copysignf(1.0f, v[i].y));
        return;
    }
    bool divide = false;
#pragma unroll
    for (int i = 0; i < N; i++) {
        t[i] = llt_sign2(v[i]);
        divide |= llt_divides2(v[i]);
    }
    if (divide)
#pragma unroll
        for (int i = 0; i < N; i++) t[i] = llt_quot2(v[i]);
}

struct LltPlan {
    dim3 grid, block;
    long long nblocks = 0;
    int zchunk = 0;
    bool pair = false;  // the two-voxels-per-thread kernel (llt_pair.cu)
};

// volumes with nx even and fewer than 2^31 voxels run k_llt_pair (3D) or
// k_llt_pair2d (CILREG_LLT_KERNEL=stream selects k_llt_stream)
bool llt_pair_applies(const Dims& d);
LltPlan llt_pair_plan(const Dims& d);
cudaError_t llt_pair_launch(const LltPlan& T, const float* cur, float* nxt, const float* f, float lam_rof,
                            float lam_llt, float tau, const Dims& d, const StopCtl* ctl, int check,
                            double2* partials, cudaStream_t s);

// 2D images run several iterations per launch (llt_strip.cu; CILREG_LLT_KERNEL
// or CILREG_STRIP2D=0 keep one per launch)
bool llt_strip_applies(const Dims& d, bool checking);
int llt_strip_run(const float* f, float* u_out, float lam_rof, float lam_llt, int iters, float tau, float epsil,
                  const Dims& d, cudaStream_t s, float* info);

}  // namespace cilreg
