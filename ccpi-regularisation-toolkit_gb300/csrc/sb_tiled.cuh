// Split-Bregman TV: the two Jacobi sweeps of one outer iteration fused into
// one 2.5D streaming kernel (sb_tiled.cu).
#pragma once

#include "drivers.cuh"
#include "pair.cuh"
#include "runtime.cuh"

namespace cilreg {

struct SbSweepArgs {
    const float* u;        // U at the start of the outer iteration
    float* u2;             // U after the second sweep
    const float* f;
    const float* dd[3];    // split variables D (read only here)
    const float* bb[3];    // Bregman variables B (read only here)
    float lambda, mu, norm;
};

// one whole outer iteration k >= 1 (k_sb_fused): D^k and B^k formed on the
// fly from U^k and B^{k-1}; writes U^{k+1} and B^k
struct SbFusedArgs {
    const float* u;        // U^k
    float* u2;             // U^{k+1}
    const float* f;
    const float* bp[3];    // B^{k-1}
    float* bn[3];          // B^k (distinct buffers: a neighbouring tile still reads B^{k-1})
    float lambda, mu, norm, dlam;
};

// D = shrink(g + b) and B = b + (g - D) of a voxel pair's N components
// (SB_TV_core.c:284-371)
template <int N>
__device__ __forceinline__ void sb_shrink2(const float2 (&g)[N], const float2 (&b)[N], float dlam, bool aniso,
                                           float2 (&dd)[N], float2 (&n)[N]) {
    using namespace pair;
    float2 v[N];
#pragma unroll
    for (int c = 0; c < N; c++) v[c] = add2(g[c], b[c]);
    if (aniso) {
        // (v / |v|) * max(|v| - 1/lambda, 0), 0 for v == 0: the same value as a sign copy
        auto one = [&](float x) { return copysignf(fmaxf(fabsf(x) - dlam, 0.f), x); };
#pragma unroll
        for (int c = 0; c < N; c++) dd[c] = make_float2(one(v[c].x), one(v[c].y));
    } else {
        float2 sq = fma2(v[0], v[0], mul2(v[1], v[1]));
        if (N > 2) sq = fma2(v[N - 1], v[N - 1], sq);
        float2 den, r;
        norm2(sq, den, r);
        const float2 m = make_float2(fmaxf(den.x - dlam, 0.f), fmaxf(den.y - dlam, 0.f));
#pragma unroll
        for (int c = 0; c < N; c++) dd[c] = mul2(m, mul2(v[c], r));
    }
#pragma unroll
    for (int c = 0; c < N; c++) n[c] = add2(b[c], sub2(g[c], dd[c]));
}

struct SbPlan {
    dim3 grid, block;
    long long nblocks = 0;
    int zchunk = 0;
    bool use = false;  // false: the per-sweep kernels of sb.cu run instead
    bool aligned = false;  // sb_pair_plan: every array is 8-byte aligned
};

SbPlan sb_sweep2_plan(const Dims& d);
// both sweeps; on a check iteration one FP64 partial of (|U2 - U1|^2, |U2|^2)
// per CTA (SbPlan::nblocks of them)
int sb_sweep2_step(const SbPlan& T, const SbSweepArgs& a, const Dims& d, const StopCtl* ctl, int check,
                   double2* partials, cudaStream_t s);
// one outer iteration k >= 1 with the shrinkage fused in (same tiling and
// partial slots as sb_sweep2_step)
int sb_fused_step(const SbPlan& T, const SbFusedArgs& a, bool aniso, const Dims& d, const StopCtl* ctl, int check,
                  double2* partials, cudaStream_t s);

// one outer iteration k >= 1 of a 3D volume with two voxels per thread
// (sb_pair.cu); its plan's `use` is false where k_sb_fused runs instead.
// `aligned`: the caller's arrays (f, U, a session's B) are 8-byte aligned
SbPlan sb_pair_plan(const Dims& d, bool aligned);
int sb_pair_step(const SbPlan& T, const SbFusedArgs& a, bool aniso, const Dims& d, const StopCtl* ctl, int check,
                 double2* partials, cudaStream_t s);

// 2D images run several outer iterations per launch (sb_strip.cu;
// CILREG_SB_KERNEL or CILREG_STRIP2D=0 keep one per launch).  `in` brings f and
// the scalars; with `warm`, iteration 0 takes its D and B, which become those
// after the n iterations run
bool sb_strip_applies(const Dims& d);
int sb_strip_run(const SbSweepArgs& in, float dlam, bool aniso, float* u_out, int iters, float epsil, const Dims& d,
                 cudaStream_t s, float* info, SbWarm* warm);

// D^n and B^n of an image from its U^n and the B^{n-1} in warm.bb, in place (sb.cu)
int sb_shrink2d(const SbSweepArgs& in, float dlam, bool aniso, const float* u, const SbWarm& warm, const Dims& d,
                const StopCtl* ctl, cudaStream_t s);

}  // namespace cilreg
