// Host runtime shared by all regulariser drivers: error reporting, per-thread
// streams, stream-ordered scratch allocation and the device-side stopping
// control.  Nothing here synchronises the device per iteration.
#pragma once

#include <stdlib.h>

#include <cuda_runtime.h>
#include <stdint.h>
#include <stddef.h>

#include "common.cuh"
#include "nvtx.cuh"

namespace cilreg {

// status codes returned through the C ABI (0 = success, negative = failure,
// the sign convention of the reference's shared.h:15-38)
enum Status : int {
    OK = 0,
    ERR_CUDA = -1,
    ERR_ARG = -2,
    ERR_NODEV = -3,
    ERR_OOM = -4,
    ERR_CANCELLED = -5,
};

// Host-side fault injection for tests: the next `n` device allocations the
// library makes (scratch and prox sessions) fail as if the device were full.
void inject_allocation_failures(int n);
// true (and one fewer pending failure) when an injected failure is due
bool take_injected_failure();

// record an error (thread-local message, also printed to stderr like the
// reference's CHECK macro) and return the status
int fail(int status, const char* file, int line, const char* fmt, ...);
const char* last_error();

#define CILREG_CUDA(call)                                                                         \
    do {                                                                                          \
        cudaError_t e_ = (call);                                                                  \
        if (e_ != cudaSuccess)                                                                    \
            return ::cilreg::fail(e_ == cudaErrorMemoryAllocation ? ::cilreg::ERR_OOM             \
                                                                   : ::cilreg::ERR_CUDA,          \
                                  __FILE__, __LINE__, "code: %d, reason: %s", (int)e_,            \
                                  cudaGetErrorString(e_));                                        \
    } while (0)

#define CILREG_TRY(expr)          \
    do {                          \
        int s_ = (expr);          \
        if (s_ != 0) return s_;   \
    } while (0)

// select the device (checks that one exists) and prepare its memory pool
int use_device(int dev);

// wait for the device's work, then return the memory its pool holds unused
int release_cached(int dev);

// a non-blocking stream owned by the calling host thread for device `dev`
cudaStream_t thread_stream(int dev);

// number of SMs of the current device (cached per device)
int sm_count();

// z-chunk length for a 2.5D streaming kernel: `tiles_xy` CTAs per z chunk,
// `resident` CTAs per SM, `extra` pipeline steps per chunk besides its planes,
// up to `max_chunk` planes.  Minimises (steps per CTA) x (time of a step):
//   busy > 0, and chunks of 8 planes make at most `waves` waves of CTAs: a step
//     takes as long as the CTAs that share an SM, at least `busy` of them
//     (below that, latency), need to issue it: max(busy, ceil(CTAs / SMs)).
//     Of chunks from 4 to 64 planes on nine volumes from 64^3 to 256^3 this
//     picks one within 1.3-4% of the fastest (ROF, NDF, Diff4th, LLT-ROF, FGP,
//     PD; with the late trigger 96^3 ROF 13.8 -> 9.7, FGP 12.7 -> 10.1 us).
//   otherwise: rounds of CTAs over the SMs' slots.  Above two waves the first
//     model costs up to 14% (FGP 256^3 133 against 115 us), Diff4th alone
//     gains from it throughout (512^3 704 -> 680 us).
int wave_zchunk(long long tiles_xy, int nz, int resident, int extra, int max_chunk, double busy = 0.0,
                double waves = 2.0);

// CTAs of `kernel` resident per SM at `threads` threads and no dynamic shared
// memory (at least 1)
template <class K>
int resident_ctas(K kernel, int threads) {
    int r = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r, kernel, threads, 0) != cudaSuccess || r <= 0) r = 1;
    return r;
}

// Let the current device's pool keep up to 2 GiB of freed scratch (calls on host
// arrays, use_device, keep all of it).  A pool that keeps none hands its memory
// back at every synchronisation and maps it anew in the next call: 0.2 ms on a
// 512^2 image, 1.5 ms on 43 M voxels of scratch.  cilreg_release_cached and a
// failed allocation give it back.
void retain_scratch();

// stream-ordered scratch buffers freed when the object is destroyed
class Scratch {
public:
    explicit Scratch(cudaStream_t s) : stream_(s) { retain_scratch(); }
    ~Scratch();
    // allocate `count` floats (64-byte aligned); returns nullptr on failure
    float* floats(long long count);
    void* bytes(size_t n);
    int status() const { return status_; }

private:
    static const int kMax = 1024;
    cudaStream_t stream_;
    void* ptrs_[kMax] = {};
    int n_ = 0;
    int status_ = 0;
};

// What the host sees of a run's stopping control: a copy that the finalize
// kernel of every check writes into page-locked memory, and that check's
// number, written after it.
struct StopMirror {
    StopCtl ctl;
    int seq;
};

// One check to reduce: its partials (n = 0: none) and where the rule's outcome goes.
struct Finalize {
    const double2* part;
    long long n;
    StopCtl* ctl;
    float epsil;
    int it;              // the check's iteration
    StopMirror* mirror;  // may be null
    int seq;             // the check's number, from 1; 0: not numbered
};

// Device-resident stopping control for one regulariser run.
class IterControl {
public:
    // partial_sets: 2 for runs that fold their checks
    IterControl(cudaStream_t s, Scratch& scratch, int iter_total, float epsil, long long max_partials,
                int partial_sets = 1);
    ~IterControl();
    int status() const { return status_; }
    StopCtl* ctl() const { return d_ctl_; }
    double2* partials() const { return d_part_; }
    bool checking() const { return epsil_ != 0.0f; }
    // the reference's test: a check happens at iteration `it` when it % 5 == 0
    bool is_check(int it) const { return epsil_ != 0.0f && (it % 5) == 0; }
    // enqueue the reduction of `nparts` partials for iteration `it`
    int after_check(int it, long long nparts, int k = 0);
    // the same check as an argument for the next launch, one CTA of which
    // runs it (finalize_check) beside that launch's own work; launch k's
    // partials then lie in slot k & 1
    Finalize fold_check(int it, long long nparts, int k);
    double2* partials(int k) const { return d_part_ ? d_part_ + (k & 1) * slots_ : nullptr; }
    // true when the host may stop enqueueing (the rule has fired on device)
    bool host_should_stop();
    // wait for completion and fill infovector[0..1] (host pointer, may be null)
    int finish(float* infovector, StopCtl* out = nullptr);

private:
    cudaStream_t stream_;
    StopCtl* d_ctl_ = nullptr;
    double2* d_part_ = nullptr;
    StopMirror* h_ = nullptr;  // page-locked, written by the device
    int checks_ = 0;           // checks enqueued
    long long slots_ = 0;
    int iter_total_;
    float epsil_;
    int status_ = 0;
};

// 1-D helper: grid for n elements with 256-thread CTAs
inline dim3 grid1(long long n) {
    long long b = (n + 255) / 256;
    if (b > 2147483647LL) b = 2147483647LL;
    return dim3((unsigned)(b < 1 ? 1 : b));
}

// Fixed-count iteration loops on small volumes, where a launch costs about as
// much as the kernel: enqueue(it, stream, in_graph) for it in [0, iters),
// with iterations [0, G) captured once into a CUDA graph (in_graph true; then
// tail(stream), which may advance device-side iteration state) and the graph
// replayed while G or more remain, the rest launched directly, all on this
// thread's own stream joined to `s` by events.  Only for loops whose launches
// depend on `it` through `it mod G` (G even) or on device-side state.
struct NoTail {
    int operator()(cudaStream_t) const { return 0; }
};
template <class Enq, class Tail = NoTail>
int run_replayed(int iters, int G, cudaStream_t s, Enq enqueue, Tail tail = Tail());

// Programmatic dependent launch: an iteration kernel launched with
// launch_pdl may be scheduled while the kernel before it in the stream is
// still draining; it runs pdl_wait() before its first access to anything that
// a kernel of the run writes (the previous grid has then completed and its
// writes are visible, so both the read-after-write and the write-after-read
// order of ping-pong buffers hold) and pdl_trigger() to let its own successor
// be scheduled early.  Both instructions do nothing in a kernel launched
// without the attribute.
//
// Some 2D kernels load the run's constant inputs (f, the lambda map, dTV's unit
// gradient) before pdl_wait().  That is only in order when something of the run
// already lies between the caller's last kernel and this launch: a caller's
// kernel may have triggered its dependents while it still writes f, and even one
// that never triggers is only sure to be seen after the wait.  So the first such
// launch of a run either follows a copy or a memset of the run (which the stream
// orders in full) or is launched without the attribute (launch_chained with
// follows = false).
//
// CILREG_PDL=0 launches normally (A/B checks).  Both functions return the launch
// status and clear it from the thread's error state.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
// Where a streaming kernel triggers.  At its start, the next grid's CTAs take
// the slots that this grid leaves free and wait in them, unevenly: the SMs
// with fewest of this grid's CTAs get most of the next's, and a grid of one or
// two CTAs per SM then runs three or four on some (ROF 96^3 14.2 us per
// iteration; 11.8 with the trigger after a CTA's last plane).  A grid of many
// waves leaves no free slots and gains from the early start (ROF 512^3 436
// against 448 us).
// Read anew at each use (volatile): held in a register over the plane loop, the
// answer cost D4's kernel 5%.
__device__ __forceinline__ bool pdl_many_waves() {
    unsigned x, y, z;
    asm volatile("mov.u32 %0, %%nctaid.x;\n\tmov.u32 %1, %%nctaid.y;\n\tmov.u32 %2, %%nctaid.z;" : "=r"(x), "=r"(y), "=r"(z));
    return x * y * z >= 4096u;
}
bool pdl_enabled();
// follows: the stream's last work is a kernel of the same run
template <typename... KArgs, typename... Args>
cudaError_t launch_chained(bool follows, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                           Args... args) {
    if (!follows || !pdl_enabled()) {
        kernel<<<grid, block, smem, s>>>(args...);
        return cudaGetLastError();
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1] = {};
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, ((KArgs)args)...);
    cudaGetLastError();  // the status is returned; leave no stale error behind
    return e;
}
template <typename... KArgs, typename... Args>
cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                       Args... args) {
    return launch_chained(true, kernel, grid, block, smem, s, args...);
}

// Deterministic reduction of a check's FP64 partials by one CTA of THREADS
// threads (a fixed assignment of partials to threads), then the stopping rule
// and the host's copy of it, written here instead of by a copy and an event
// per check, which kept the next iteration from starting for about 10 us.
template <int THREADS>
__device__ __forceinline__ void finalize_check(const Finalize& f) {
    if (f.ctl->stop) return;
    const int tid = threadIdx.x + blockDim.x * threadIdx.y;
    double a = 0.0, b = 0.0;
    for (long long p = tid; p < f.n; p += THREADS) {
        const double2 v = f.part[p];
        a += v.x;
        b += v.y;
    }
    __shared__ double sa[32], sb[32];
    a = warp_sum(a);
    b = warp_sum(b);
    if ((tid & 31) == 0) { sa[tid >> 5] = a; sb[tid >> 5] = b; }
    __syncthreads();
    if (tid < 32) {
        a = warp_sum(tid < THREADS / 32 ? sa[tid] : 0.0);
        b = warp_sum(tid < THREADS / 32 ? sb[tid] : 0.0);
        if (tid == 0) {
            const float re = sqrtf((float)a) / sqrtf((float)b);
            StopCtl c = *f.ctl;
            c.re = re;
            if (re < f.epsil) c.count += 1;
            if (c.count > 3) {
                c.stop = f.seq > 0 ? f.seq : 1;
                c.iters = f.it;
            }
            f.ctl->re = c.re;
            f.ctl->count = c.count;
            f.ctl->iters = c.iters;
            *(volatile int*)&f.ctl->stop = c.stop;  // other CTAs of the launch may be reading it
            if (f.mirror) {
                *(volatile int*)&f.mirror->ctl.stop = c.stop;
                *(volatile int*)&f.mirror->ctl.iters = c.iters;
                *(volatile int*)&f.mirror->ctl.count = c.count;
                *(volatile float*)&f.mirror->ctl.re = c.re;
                asm volatile("st.release.sys.global.b32 [%0], %1;" ::"l"(&f.mirror->seq), "r"(f.seq) : "memory");
            }
        }
    }
}

// process-wide count of kernels this library has launched (for benchmarks)
void note_launch(long long n = 1);
long long launch_count();

// device kernels shared by the drivers (runtime.cu)
// reset a StopCtl (no stop, iters = iter_total, count 0, re 0)
int launch_init_ctl(StopCtl* ctl, int iter_total, cudaStream_t s);
// reduce `nparts` FP64 partials and apply the stopping rule for iteration `it`
int launch_finalize_check(const double2* partials, long long nparts, StopCtl* ctl, float epsil, int it,
                          cudaStream_t s);
// per-volume stopping checks of a batch: slot v reduces part[v][0..n[v]) into ctl[v]
struct CheckSlot {
    const double2* part;
    long long n;
    StopCtl* ctl;
};
int launch_finalize_batch(const CheckSlot* d_slots, int nvol, float epsil, int it, cudaStream_t s);
int launch_init_ctls(StopCtl* const* d_ctls, int nvol, int iter_total, cudaStream_t s);
int launch_fill(float* p, float v, long long n, cudaStream_t s);
int launch_copy(float* dst, const float* src, long long n, cudaStream_t s);
// copy the buffer that holds the final iterate into dst, choosing on device:
// the last written iteration is ctl->iters when stopped, else iter_total-1;
// buffer bufs[(last+1) & 1] holds it (ping-pong with iteration it writing bufs[(it+1)&1]).
int launch_select_pingpong(const StopCtl* ctl, int iter_total, float* const bufs[2], float* dst, long long n,
                           cudaStream_t s);
// The same for runs of several iterations per launch (strip2d.cuh): launch k
// wrote src[k & 1]; the result is that of the launch whose check fired, else of
// launch `last` (nothing to copy where it lies in dst already).
struct SpanResult {
    const float* src[2];
    float* dst;
    bool stopped_only;  // dst is right already unless the rule fired
};
int launch_take_span(const StopCtl* ctl, int last, const SpanResult* results, int count, long long n, cudaStream_t s);


template <class Enq, class Tail>
int run_replayed(int iters, int G, cudaStream_t s, Enq enqueue, Tail tail) {
    CILREG_RANGE("cilreg graph replay");
    const char* env = getenv("CILREG_GRAPH_REPLAY");  // "0": launch every iteration directly (A/B checks)
    const int reps = (G > 0 && (G % 2) == 0 && !(env && env[0] == '0')) ? iters / G : 0;
    // a stream the caller is capturing records the launches as they are
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    const bool capturing = cudaStreamIsCapturing(s, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone;
    cudaGetLastError();
    if (reps < 2 || capturing) {
        for (int it = 0; it < iters; it++) CILREG_TRY(enqueue(it, s, false));
        return OK;
    }
    // capture and replay on this thread's own stream t (the caller's may be a
    // default stream, which cannot be captured), ordered after the caller's
    // earlier work and before its later work by two events
    int dev = 0;
    CILREG_CUDA(cudaGetDevice(&dev));
    cudaStream_t t = thread_stream(dev);
    cudaEvent_t ev[2] = {nullptr, nullptr};
    for (int i = 0; i < 2; i++) CILREG_CUDA(cudaEventCreateWithFlags(&ev[i], cudaEventDisableTiming));
    auto finish = [&](int rc) {
        for (int i = 0; i < 2; i++) cudaEventDestroy(ev[i]);
        return rc;
    };
    if (t != s) {
        if (cudaEventRecord(ev[0], s) != cudaSuccess || cudaStreamWaitEvent(t, ev[0], 0) != cudaSuccess)
            return finish(fail(ERR_CUDA, __FILE__, __LINE__, "stream ordering failed"));
    }
    cudaGraph_t g = nullptr;
    cudaGraphExec_t ge = nullptr;
    if (cudaStreamBeginCapture(t, cudaStreamCaptureModeThreadLocal) != cudaSuccess)
        return finish(fail(ERR_CUDA, __FILE__, __LINE__, "stream capture failed"));
    const long long before = launch_count();
    int rc = OK;
    for (int k = 0; k < G && rc == OK; k++) rc = enqueue(k, t, true);
    if (rc == OK) rc = tail(t);
    const cudaError_t e = cudaStreamEndCapture(t, &g);
    if (rc != OK) {
        if (g) cudaGraphDestroy(g);
        return finish(rc);
    }
    if (e != cudaSuccess) return finish(fail(ERR_CUDA, __FILE__, __LINE__, "%s", cudaGetErrorString(e)));
    const cudaError_t ei = cudaGraphInstantiate(&ge, g, 0);
    cudaGraphDestroy(g);
    if (ei != cudaSuccess) return finish(fail(ERR_CUDA, __FILE__, __LINE__, "%s", cudaGetErrorString(ei)));
    const long long per_graph = launch_count() - before;
    cudaError_t el = cudaSuccess;
    for (int r = 0; r < reps && el == cudaSuccess; r++) el = cudaGraphLaunch(ge, t);
    cudaGraphExecDestroy(ge);  // freed when the queued launches complete
    if (el != cudaSuccess) return finish(fail(ERR_CUDA, __FILE__, __LINE__, "%s", cudaGetErrorString(el)));
    note_launch(per_graph * (reps - 1));  // the capture counted one replay
    for (int it = reps * G; it < iters && rc == OK; it++) rc = enqueue(it, t, false);
    if (rc != OK) return finish(rc);
    if (t != s) {
        if (cudaEventRecord(ev[1], t) != cudaSuccess || cudaStreamWaitEvent(s, ev[1], 0) != cudaSuccess)
            return finish(fail(ERR_CUDA, __FILE__, __LINE__, "stream ordering failed"));
    }
    return finish(OK);
}


}  // namespace cilreg
