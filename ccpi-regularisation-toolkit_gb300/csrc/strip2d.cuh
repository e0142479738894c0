// 2D images, several iterations per launch: the tile scheme shared by the
// strip kernels.
//
// What bounds a 2D iteration launched by itself is not its bytes or its
// arithmetic but the launch: a 512^2 image's iteration takes 0.1-0.3 us of
// the chip's issue slots and 2.4-4 us as a graph node.  A strip kernel loads
// a tile with a halo of `margin` pixels once, runs `count` <= margin
// iterations on it and stores the part that no cut side has reached.
//
// A CTA of NW warps holds a tile of 64 x (NW R) pixels entirely in registers:
// a lane holds a pixel pair (x, x+1) of R consecutive rows, a warp whole rows
// of 64 pixels.  Then
//   * the x neighbours of a pair are its own other pixel and one shuffle;
//   * the y neighbours are the thread's own registers, except at the first
//     and last row of a strip, which every warp publishes in shared memory
//     (two slots, so one barrier per iteration suffices);
//   * what an iteration needs of a row above or below the strip (a flux, a
//     projected dual) is recomputed from the published row instead of being
//     exchanged after a second barrier.
// Pixels within t of a cut side of the tile are stale after t iterations;
// sides on the image's edge are exact (the mirrored neighbour, by selects
// that only strips at the edge execute), so the first and last tile of an
// axis have no halo on that side.
#pragma once

#include <float.h>

#include "drivers.cuh"
#include "pair.cuh"

namespace cilreg {
namespace strip {

using namespace pair;

constexpr int NW = 16;       // warps of a CTA (32 of 2 rows measured 1.2-1.5 times slower than 16 of 4)
constexpr int NT = 32 * NW;  // threads of a CTA
constexpr int SW = 64;       // tile width
constexpr int MAXT = 16;     // largest number of iterations per launch

struct Plan {
    int R = 0;       // rows per thread; 0: the image does not run strips
    int T = 0;       // most iterations per launch
    int margin = 0;  // halo of the tiles
    int gx = 0, gy = 0;  // tiles along x and y
    long long nblocks = 0;
};

// CILREG_STRIP2D=0 runs 2D images one iteration per launch; =R,T asks for R
// rows per thread and T iterations per launch where they are among the choices
// (A/B checks and tests)
bool enabled();
bool forced(int* R, int* T);

// tiles that cover n pixels: tile i starts at i (len - 2 margin), the first
// and the last reach the image's edges
inline int tiles(int n, int len, int margin) {
    const int step = len - 2 * margin;
    return n <= len ? 1 : 1 + (n - len + step - 1) / step;
}

// The rows per thread and the iterations per launch (1 .. 16; 5 with a
// stopping rule, whose checks end a launch) with the lowest modelled time per
// iteration, in cycles.  A launch costs LAUNCH and then its waves of CTAs; a
// wave costs start + R start_row (a tile's loads and stores) and lat + R
// lat_row per iteration (a warp's dependent instructions) with one CTA per SM,
// PAIRED times that with two (STEADY where CTAs replace each other as they
// end).  Fitted to ROF on images of 181x217 to 3000x2900 (within 15%); the
// other regularisers bring the constants measured on them.
struct Choices {
    int radius;       // stale pixels per iteration at a cut side
    int n;            // number of kernels
    int rows[4];      // their rows per thread
    int resident[4];  // CTAs per SM (1 or 2)
    double lat, lat_row;
    double start = 2200.0, start_row = 0.0;
};
constexpr double LAUNCH = 1500.0, PAIRED = 1.65, STEADY = 1.4;
inline Plan plan(int nx, int ny, int iters, bool checking, const Choices& c) {
    int fr = 0, ft = 0;
    const bool ask = forced(&fr, &ft);
    for (int pass = ask ? 0 : 1; pass < 2; pass++) {
        Plan best;
        double best_cost = 0.0;
        const int tmax = checking ? 5 : (iters < 1 ? 1 : (iters < MAXT ? iters : MAXT));
        for (int q = 0; q < c.n; q++) {
            const int R = c.rows[q], H = NW * R;
            if (pass == 0 && R != fr) continue;
            for (int t = checking ? 5 : 1; t <= tmax; t++) {
                const int m = t * c.radius;
                if (2 * m > SW / 2 || 2 * m > H - 14) break;  // tiles keep half their width and 14 rows
                if (pass == 0 && !checking && t != (ft < tmax ? ft : tmax)) continue;
                const long long nb = (long long)tiles(nx, SW, m) * tiles(ny, H, m);
                const double per_sm = (double)nb / sm_count();
                const int res = c.resident[q];
                const double one = c.start + R * c.start_row + t * (c.lat + R * c.lat_row);
                const double two = one * (res == 2 ? PAIRED : 1.0);
                double wait;
                if (per_sm <= 1.0)
                    wait = one;
                else if (per_sm <= 2.0 * res)
                    wait = per_sm <= res ? two : (per_sm <= 3.0 && res == 2 ? one + two : 2.0 * two);
                else
                    wait = (per_sm / res + 0.3) * one * (res == 2 ? STEADY : 1.0);
                const double cost = (LAUNCH + wait) / t;
                if (best.R == 0 || cost < best_cost) {
                    best_cost = cost;
                    best.R = R;
                    best.T = t;
                    best.margin = m;
                    best.gx = tiles(nx, SW, m);
                    best.gy = tiles(ny, H, m);
                    best.nblocks = nb;
                }
            }
        }
        if (best.R) return best;
    }
    return Plan{};
}

// What every launch gets besides its arrays: the image, the tiles, and the
// check of the launch before, which CTA 0 then reduces while the others run.
// The stop it may set holds from the launch after this one on (tile_runs), whose
// tiles then leave both launches' results alone: launch k and k+1 write different
// buffers, so a run that stops at launch k's check ends on k's.  (A finalize
// kernel between them cost 7 us per check.)  RULE: the run has a stopping rule;
// the kernels of runs without one are compiled without all of this, which
// would cost them 3 to 10%.
struct Frame {
    int nx, ny, margin, count, gx;
    bool aligned;
    bool follows;  // not the run's first launch
    const StopCtl* ctl;
    double2* partials;
    Finalize check;
};
template <bool RULE>
__device__ __forceinline__ int tile_index(const Frame& F) {
    return (int)blockIdx.x - (RULE && F.check.n > 0 ? 1 : 0);
}
// waits for the launch before; false where the CTA has no tile to run
template <bool RULE>
__device__ __forceinline__ bool begin(const Frame& F) {
    pdl_wait();
    pdl_trigger();
    if (!RULE) return true;
    if (tile_index<RULE>(F) < 0) {
        finalize_check<NT>(F.check);
        return false;
    }
    return tile_runs(*(const volatile int*)&F.ctl->stop, F.check.n > 0 ? F.check.seq : 0);
}
// Launches one launch of a run, `args` and then the frame.  The kernels load the
// run's constant inputs before pdl_wait(), so the first launch, right behind
// whatever wrote those inputs, waits for it in full like any kernel (launch_pdl).
template <class Kernel, class... Args>
cudaError_t launch_strip(Kernel kernel, const Plan& P, const Frame& F, bool rule, cudaStream_t s, Args... args) {
    const dim3 grid = rule ? dim3((unsigned)(P.nblocks + (F.check.n > 0 ? 1 : 0))) : dim3((unsigned)P.gx, (unsigned)P.gy);
    return launch_chained(F.follows, kernel, grid, dim3(32, NW, 1), 0, s, args..., F);
}
// A thread's sums of a check over its rows: squared change (x) and square (y),
// each as an FP32 sum and its rounding error, so that a thread's rows lose
// nothing to each other.  (FP64 sums instead would be 2 R additions in every
// warp, 16 cycles each.)  The two sums issue paired.
struct Norms {
    float2 s = make_float2(0.f, 0.f), e = make_float2(0.f, 0.f);
};
__device__ __forceinline__ void add_exact(Norms& n, float2 x) {
    const float2 t = add2(n.s, x), v = sub2(t, n.s);
    n.e = add2(n.e, add2(sub2(n.s, sub2(t, v)), sub2(x, v)));
    n.s = t;
}

// One FP64 partial of the CTA's sums.  Two warps add the threads' sums from
// shared memory: the FP64 unit takes 16 cycles for a warp's addition, and a
// shuffle reduction of both sums in every warp is 170 of them per CTA against
// 44.  The errors, 2^-24 of the sums, are added in FP32.
__device__ __forceinline__ void store_partial(const Norms& n, double2* slot) {
    __shared__ float sum[2][NT], err[2][NW];
    const int lane = threadIdx.x, w = threadIdx.y;
    sum[0][w * 32 + lane] = n.s.x;
    sum[1][w * 32 + lane] = n.s.y;
    float ea = fabsf(n.e.x) <= FLT_MAX ? n.e.x : 0.f, eb = fabsf(n.e.y) <= FLT_MAX ? n.e.y : 0.f;  // an infinite sum has none
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        ea += __shfl_down_sync(0xffffffffu, ea, o);
        eb += __shfl_down_sync(0xffffffffu, eb, o);
    }
    if (lane == 0) {
        err[0][w] = ea;
        err[1][w] = eb;
    }
    __syncthreads();
    if (w < 2) {
        double v = lane < NW ? (double)err[w][lane] : 0.0;
#pragma unroll
        for (int j = 0; j < NW; j++) v += (double)sum[w][j * 32 + lane];
        v = warp_sum(v);
        if (lane == 0) (w == 0 ? slot->x : slot->y) = v;
    }
}

// a thread's place in its tile and what it may store
template <int R>
struct Place {
    int lane, w;
    int X, Y;        // pixel of the thread's first voxel
    int nx, ny;
    bool vx, vy;     // columns X, X+1 are stored
    int y0, y1;      // rows [y0, y1) are stored
    bool edge;       // an end of the rows, or the last row, lies in the strip or right under it (uniform over the warp)
    bool at_left, at_right, odd_end;  // the pair starts a row; ends it; its first pixel ends it
    int bottom;      // the strip's row that is the image's last, if any
    int c0, c1;      // columns clamped into the image
    bool vec;        // 8-byte accesses
    __device__ __forceinline__ Place(const Frame& F, bool rule, int tile) : nx(F.nx), ny(F.ny) {
        constexpr int H = NW * R;
        const int margin = F.margin;
        lane = threadIdx.x;
        w = threadIdx.y;
        const int bx = rule ? tile % F.gx : blockIdx.x, by = rule ? tile / F.gx : blockIdx.y;
        const int X0 = bx * (SW - 2 * margin), Y0 = by * (H - 2 * margin);
        X = X0 + 2 * lane;
        Y = Y0 + w * R;
        const int xa = X0 ? X0 + margin : 0, xb = (X0 + SW >= nx) ? nx : X0 + SW - margin;
        y0 = Y0 ? Y0 + margin : 0;
        y1 = (Y0 + H >= ny) ? ny : Y0 + H - margin;
        vx = X >= xa && X < xb;
        vy = X + 1 >= xa && X + 1 < xb;
        edge = X0 == 0 || X0 + SW >= nx || (Y < ny && Y + R + 1 >= ny);
        at_left = X == 0;
        at_right = X + 2 == nx;
        odd_end = X + 1 == nx;
        bottom = ny - 1 - Y;
        vec = F.aligned && (nx & 1) == 0;
        c0 = vec ? min(X, nx - 2) : min(X, nx - 1);
        c1 = min(X + 1, nx - 1);
    }
    __device__ __forceinline__ int row(int r) const { return min(Y + r, ny - 1) * nx; }
    __device__ __forceinline__ float2 load_const(const float* __restrict__ p, int r) const {
        const float* q = p + row(r);
        if (vec) return __ldg(reinterpret_cast<const float2*>(q + c0));
        return make_float2(__ldg(q + c0), __ldg(q + c1));
    }
    __device__ __forceinline__ float2 load(const float* p, int r) const {
        const float* q = p + row(r);
        if (vec) return *reinterpret_cast<const float2*>(q + c0);
        return make_float2(q[c0], q[c1]);
    }
    __device__ __forceinline__ void store(float* p, int r, float2 v) const {
        const int y = Y + r;
        if (y < y0 || y >= y1) return;
        float* q = p + (y * nx + X);
        if (vec && vx && vy) {
            st2(q, v);
        } else {
            if (vx) q[0] = v.x;
            if (vy) q[1] = v.y;
        }
    }
};

// 1/sqrt(s) for normal s: the flush-to-zero form of rsqrtf's approximation,
// the same value without the scaling that subnormal arguments need
__device__ __forceinline__ float rsqrt_normal(float s) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(s));
    return r;
}

// the pixel left of a pair's first and right of its second, from the
// neighbouring lanes (the tile's outermost lanes get their own pixel back)
__device__ __forceinline__ float left_of(float2 v) { return __shfl_up_sync(0xffffffffu, v.y, 1); }
__device__ __forceinline__ float right_of(float2 v) { return __shfl_down_sync(0xffffffffu, v.x, 1); }

// The launches of a run: iterations [first, first + count) each; with a
// stopping rule every check iteration (0, 5, 10, ...) ends a launch.
struct Span {
    int first, count;
    bool check;
};
template <class F>
int for_spans(int iters, int most, bool checking, F f) {
    int it = 0, k = 0;
    while (it < iters) {
        int n = checking ? (it == 0 ? 1 : 5) : most;
        if (n > iters - it) n = iters - it;
        const Span s{it, n, checking && (it + n - 1) % 5 == 0};
        const int rc = f(k, s);
        if (rc != 0) return rc < 0 ? rc : 0;
        it += n;
        k++;
    }
    return 0;
}
inline int count_spans(int iters, int most, bool checking) {
    if (iters <= 0) return 0;
    return checking ? 1 + (iters - 1 + 4) / 5 : (iters + most - 1) / most;
}
// index of the launch that runs check iteration `it`
__host__ __device__ inline int span_of_check(int it) { return it / 5; }

// the images that strips take
inline bool applies(const Dims& d) { return d.nz == 1 && d.nx > 1 && d.ny > 1 && d.n < (1LL << 31) && enabled(); }

// an x neighbour pair of v: (x-1, x) and (x+1, x+2), mirrored at the ends of
// the image's rows; the pixel beyond an odd row takes its mirrored value
template <bool EDGE, int R>
__device__ __forceinline__ void x_neighbours(const Place<R>& q, float2& v, float& lo, float& hi) {
    lo = left_of(v);
    hi = right_of(v);
    if (EDGE) {
        if (q.odd_end) v.y = lo;
        if (q.at_left) lo = v.y;
        if (q.at_right) hi = v.x;
    }
}

// A launch's iterations: pass(t, last).  With a rule the last one, whose change a
// check sums, is a copy of its own, so that the sums take no registers before it
// (a type, not a bool, as `last`).
template <bool B>
struct Flag {
    __device__ constexpr operator bool() const { return B; }
};
template <bool CHECK, class Pass>
__device__ __forceinline__ void iterations(int count, Pass pass) {
    if constexpr (CHECK) {
        for (int t = 0; t < count - 1; t++) pass(t, Flag<false>{});
        pass(count - 1, Flag<true>{});
    } else {
        for (int t = 0; t < count; t++) pass(t, t == count - 1);
    }
}

// adds the stored pixels' squared change and square of one row
template <int R>
__device__ __forceinline__ void add_norms(const Place<R>& q, int r, float2 un, float2 u, Norms& n) {
    if (q.Y + r < q.y0 || q.Y + r >= q.y1) return;
    const float2 df = sub2(un, u);
    const float2 dm = make_float2(q.vx ? df.x : 0.f, q.vy ? df.y : 0.f);
    const float2 um = make_float2(q.vx ? un.x : 0.f, q.vy ? un.y : 0.f);
    // as the kernels of one iteration per launch: a pixel pair of even rows summed
    // in FP32, every pixel of odd rows by itself
    const float2 x = make_float2(dm.x, um.x), y = make_float2(dm.y, um.y);
    if (q.nx & 1) {
        add_exact(n, mul2_rn(x, x));
        add_exact(n, mul2_rn(y, y));
    } else {
        add_exact(n, fma2(y, y, mul2_rn(x, x)));
    }
}

// The launches of a run: each(k, span, frame) enqueues launch k.  The check of
// launch k rides on launch k+1, the last launch's gets a kernel of its own.
template <class F>
int run_spans(const Plan& P, IterControl& ctl, int iters, bool checking, const Dims& d, bool aligned, F each) {
    const int nl = count_spans(iters, P.T, checking);
    Finalize pending = {};
    return for_spans(iters, P.T, checking, [&](int k, const Span& sp) -> int {
        const Frame fr{d.nx,  d.ny,      P.margin,        sp.count, P.gx,
                       aligned, k > 0, ctl.ctl(), ctl.partials(k), pending};
        CILREG_TRY(each(k, sp, fr));
        note_launch();
        pending = Finalize{};
        if (!sp.check) return 0;
        const int it = sp.first + sp.count - 1;
        if (k == nl - 1) return ctl.after_check(it, P.nblocks, k);
        pending = ctl.fold_check(it, P.nblocks, k);
        return ctl.host_should_stop() ? 1 : 0;
    });
}

// U of a run whose launch k writes bufs[(nl - 1 - k) & 1]
inline SpanResult span_result(float* const bufs[2], int nl, float* dst) {
    return SpanResult{{bufs[(nl - 1) & 1], bufs[nl & 1]}, dst, false};
}

// The run of a regulariser whose state is one image U beside f (ROF, NDF,
// Diff4th, LLT-ROF): launch(plan, rule, frame, src, dst) enqueues one launch.
// Launch k writes bufs[(nl - 1 - k) & 1], so the last writes u_out; a run that
// stops early on the other buffer copies it.  The copy is chosen on the device
// and enqueued before the call waits for the stream: the output is complete when
// the call returns.
template <class Launch>
int run_flow(const Choices& choices, const float* f, const float* start, float* u_out, int iters, float epsil,
             const Dims& d, cudaStream_t s, float* info, bool aligned, Launch launch) {
    const bool checking = epsil != 0.0f;
    const Plan P = plan(d.nx, d.ny, iters, checking, choices);
    Scratch scratch(s);
    IterControl ctl(s, scratch, iters, epsil, P.nblocks, 2);
    CILREG_TRY(ctl.status());
    const size_t bytes = sizeof(float) * (size_t)d.n;
    if (iters <= 0) CILREG_CUDA(cudaMemcpyAsync(u_out, start, bytes, cudaMemcpyDeviceToDevice, s));
    const int nl = count_spans(iters, P.T, checking);
    float* alt = nl > 1 ? scratch.floats(d.n) : nullptr;
    if (nl > 1 && !alt) return scratch.status();
    float* bufs[2] = {u_out, alt};
    aligned = aligned && host_aligned8(f) && host_aligned8(start) && host_aligned8(u_out);
    CILREG_TRY(run_spans(P, ctl, iters, checking, d, aligned, [&](int k, const Span&, const Frame& fr) -> int {
        CILREG_CUDA(launch(P, checking, fr, k == 0 ? start : bufs[(nl - k) & 1], bufs[(nl - 1 - k) & 1]));
        return OK;
    }));
    if (checking && nl > 1) {
        const SpanResult r = span_result(bufs, nl, u_out);
        CILREG_TRY(launch_take_span(ctl.ctl(), nl - 1, &r, 1, d.n, s));
    }
    return ctl.finish(info);
}

}  // namespace strip
}  // namespace cilreg
