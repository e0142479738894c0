// 2.5D streaming fourth-order diffusion iteration (diff4th_tiled.cu).
#pragma once

#include "runtime.cuh"

namespace cilreg {

struct D4Plan {
    dim3 grid, block;
    long long nblocks = 0;
    int zchunk = 0;
    bool pair = false;  // the two-voxels-per-thread kernel (diff4th_pair.cu)
};

// the plan of the streaming kernel that runs for `d`: with `pairs`, volumes of fewer than
// 2^31 voxels (rows of two voxels, or three and more) run k_d4_pair, images with
// nx even k_d4_pair2d where they do not run strips (CILREG_D4_KERNEL=stream
// selects k_d4_stream), others k_d4_stream
D4Plan d4_stream_plan(const Dims& d, bool pairs);
bool d4_pair_applies(const Dims& d);
D4Plan d4_pair_plan(const Dims& d);
int d4_pair_step(const D4Plan& T, const float* cur, float* nxt, const float* f, float lam, float tau, float isg2,
                 const Dims& d, const StopCtl* ctl, int check, double2* partials, cudaStream_t s);
// 2D images run several iterations per launch (diff4th_strip.cu;
// CILREG_D4_KERNEL or CILREG_STRIP2D=0 keep one per launch)
bool d4_strip_applies(const Dims& d);
int d4_strip_run(const float* f, float* u_out, float lam, int iters, float tau, float isg2, float epsil, const Dims& d,
                 cudaStream_t s, float* info);
// one iteration: reads cur, writes nxt (distinct buffers); isg2 = 1/sigma^2
int d4_stream_step(const D4Plan& T, const float* cur, float* nxt, const float* f, float lam, float tau, float isg2,
                   const Dims& d, const StopCtl* ctl, int check, double2* partials, cudaStream_t s);

}  // namespace cilreg
