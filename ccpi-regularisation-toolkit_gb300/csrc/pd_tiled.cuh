// 2.5D streaming PD-TV iteration (pd_tiled.cu).
#pragma once

#include "pd_math.cuh"
#include "runtime.cuh"

namespace cilreg {

struct PdStreamArgs {
    const float* u;     // extrapolated primal iterate Ue (current)
    float* un;          // Ue (next)
    const float* p[3];  // dual (current)
    float* pn[3];       // dual (next)
    const float* f;
    float* ubrk;        // U before extrapolation, written on check iterations
    float sigma, tau, lt, theta;
    DoubleDivisor onelt;  // the reference's double (1.0 + lt)
    int nonneg, aniso, check;
};

struct PdPlan {
    dim3 grid, block;
    long long nblocks = 0;
    int zchunk = 0;
    bool pair = false;     // two voxels per thread (pd_pair.cu)
    bool aligned = false;  // of pair: every array is 8-byte aligned
};

PdPlan pd_stream_plan(const Dims& d);
int pd_stream_step(const PdPlan& T, const PdStreamArgs& a, const Dims& d, const StopCtl* ctl, double2* partials,
                   cudaStream_t s);

// one iteration of a 3D volume with two voxels per thread (pd_pair.cu);
// `aligned`: the caller's arrays (f, U) are 8-byte aligned
PdPlan pd_pair_plan(const Dims& d, bool aligned);
int pd_pair_step(const PdPlan& T, const PdStreamArgs& a, const Dims& d, const StopCtl* ctl, double2* partials,
                 cudaStream_t s);

// 2D images run several iterations per launch (pd_strip.cu; CILREG_PD_KERNEL or
// CILREG_STRIP2D=0 keep one per launch)
bool pd_strip_applies(const Dims& d);
int pd_strip_run(const float* f, float* u_out, float sigma, float tau, float lt, const DoubleDivisor& onelt, int iters,
                 float epsil, bool nonneg, bool aniso, const Dims& d, cudaStream_t s, float* info);

}  // namespace cilreg
