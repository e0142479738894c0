// TGV on 2D images, several iterations per launch (strip2d.cuh) with U, V, P
// and Q of a thread's pixels in registers (TGV_core.c:43-345).  The dual half
// of an iteration needs U and V of the row under a strip, the primal half P
// and Q of the row above it: each is published before the half that needs it.
#include <algorithm>

#include <float.h>

#include "strip2d.cuh"
#include "tgv_tiled.cuh"

namespace cilreg {

namespace {

using namespace strip;

constexpr int NS = 7;  // V1 V2 P1 P2 Q1 Q2 Q3

struct Args {
    const float* u;
    float* un;
    const float* s[NS];  // null: zero
    float* sn[NS];       // null: not stored
    const float* f;
    float tau, lambda, inv_lt, alpha1, alpha0, near1, near0;
};

// 1 / (sqrt(s) / alpha) where sqrt(s) / alpha > 1, else 1 (ProjP, ProjQ: TGV_core.c:221-231,
// 262-274).  `near` lies just under alpha^2: below it the quotient is under 1
// and the root and the division are skipped.
__device__ __forceinline__ float2 ball_scale(float2 s, float alpha, float near) {
    float2 ig = splat(1.f);
    if (s.x > near || s.y > near) {
        const float gx = sqrtf(s.x) / alpha, gy = sqrtf(s.y) / alpha;
        if (gx > 1.0f) ig.x = __frcp_rn(gx);
        if (gy > 1.0f) ig.y = __frcp_rn(gy);
    }
    return ig;
}

template <int R, bool CHECK>
__global__ void __launch_bounds__(NT, 1) k_tgv_strip2d(Args a, Frame fr) {
    __shared__ float2 firstUV[3][NW][32], lastPQ[3][NW][32];
    const Place<R> q(fr, CHECK, max(tile_index<CHECK>(fr), 0));
    const int lane = q.lane, w = q.w;
    float2 tf[R];
#pragma unroll
    for (int r = 0; r < R; r++) tf[r] = mul2(splat(a.tau), q.load_const(a.f, r));  // never changes: before the wait
    if (!begin<CHECK>(fr)) return;
    float2 u[R], v1[R], v2[R], p1[R], p2[R], q1[R], q2[R], q3[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
        u[r] = q.load(a.u, r);
        v1[r] = v2[r] = p1[r] = p2[r] = q1[r] = q2[r] = q3[r] = splat(0.f);
    }
    if (a.s[0]) {
#pragma unroll
        for (int r = 0; r < R; r++) {
            v1[r] = q.load(a.s[0], r);
            v2[r] = q.load(a.s[1], r);
            p1[r] = q.load(a.s[2], r);
            p2[r] = q.load(a.s[3], r);
            q1[r] = q.load(a.s[4], r);
            q2[r] = q.load(a.s[5], r);
            q3[r] = q.load(a.s[6], r);
        }
    }
    const float2 tau2 = splat(a.tau), lam2 = splat(a.lambda), ilt2 = splat(a.inv_lt), HALF2 = splat(0.5f),
                 TWO2 = splat(2.f);
    Norms norms;

    // P and Q (sigma == tau)
    auto dual = [&](auto edge_, float2 ub, float2 v1b, float2 v2b) {
        constexpr bool EDGE = decltype(edge_)::value;
        // difference to the next pixel, 0 at the last index
        auto ahead_x = [&](float2 c) {
            float2 e = make_float2(c.y - c.x, right_of(c) - c.y);
            if (EDGE) {
                if (q.at_right) e.y = 0.f;
                if (q.odd_end) e.x = 0.f;
            }
            return e;
        };
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int n = r + 1 < R ? r + 1 : r;
            const bool lastrow = EDGE && r == q.bottom;
            auto ahead_y = [&](float2 next, float2 c) { return lastrow ? splat(0.f) : sub2(next, c); };
            const float2 uy = ahead_y(r + 1 < R ? u[n] : ub, u[r]);
            const float2 y1 = ahead_y(r + 1 < R ? v1[n] : v1b, v1[r]), y2 = ahead_y(r + 1 < R ? v2[n] : v2b, v2[r]);
            // DualP_2D + ProjP_2D (TGV_core.c:200-232)
            float2 a1 = fma2(tau2, sub2(ahead_x(u[r]), v1[r]), p1[r]);
            float2 a2 = fma2(tau2, sub2(uy, v2[r]), p2[r]);
            const float2 ip = ball_scale(fma2(a1, a1, mul2(a2, a2)), a.alpha1, a.near1);
            p1[r] = mul2(a1, ip);
            p2[r] = mul2(a2, ip);
            // DualQ_2D + ProjQ_2D (TGV_core.c:234-275)
            const float2 x1 = ahead_x(v1[r]), x2 = ahead_x(v2[r]);
            const float2 b1 = fma2(tau2, x1, q1[r]), b2 = fma2(tau2, y2, q2[r]);
            const float2 b3 = fma2(tau2, mul2(HALF2, add2(x2, y1)), q3[r]);
            const float2 iq =
                ball_scale(fma2(mul2(TWO2, b3), b3, fma2(b1, b1, mul2(b2, b2))), a.alpha0, a.near0);
            q1[r] = mul2(b1, iq);
            q2[r] = mul2(b2, iq);
            q3[r] = mul2(b3, iq);
        }
    };
    // U and V; (p2u, q2u, q3u): P2, Q2, Q3 of the row above
    auto primal = [&](auto edge_, float2 p2u, float2 q2u, float2 q3u, auto sum) {
        constexpr bool EDGE = decltype(edge_)::value;
        // backward differences: X at index 0, -X[-1] at the last (TGV_core.c:286-292)
        auto back_x = [&](float2 c) {
            float lo = left_of(c);
            if (EDGE && q.at_left) lo = 0.f;
            float2 e = make_float2(c.x - lo, c.y - c.x);
            if (EDGE) {
                if (q.at_right) e.y = -c.x;
                if (q.odd_end) e.x = -lo;
            }
            return e;
        };
#pragma unroll
        for (int r = 0; r < R; r++) {
            const bool lastrow = EDGE && r == q.bottom;
            auto back_y = [&](float2 c, float2 up) { return lastrow ? neg2(up) : sub2(c, up); };
            // DivProjP_2D + newU (TGV_core.c:277-306)
            const float2 dv = add2(back_x(p1[r]), back_y(p2[r], p2u));
            const float2 un = mul2(fma2(lam2, fma2(tau2, dv, u[r]), tf[r]), ilt2);
            const float2 ue = fma2(TWO2, un, neg2(u[r]));
            if (CHECK && sum) add_norms(q, r, ue, u[r], norms);
            u[r] = ue;
            // UpdV_2D + newV (TGV_core.c:308-345)
            const float2 d1 = add2(back_x(q1[r]), back_y(q3[r], q3u));
            const float2 d2 = add2(back_x(q3[r]), back_y(q2[r], q2u));
            v1[r] = fma2(TWO2, fma2(tau2, add2(p1[r], d1), v1[r]), neg2(v1[r]));
            v2[r] = fma2(TWO2, fma2(tau2, add2(p2[r], d2), v2[r]), neg2(v2[r]));
            p2u = p2[r];
            q2u = q2[r];
            q3u = q3[r];
        }
    };
    const bool top = q.Y == 0;
    iterations<CHECK>(fr.count, [&](int t, auto sum) {
        firstUV[0][w][lane] = u[0];
        firstUV[1][w][lane] = v1[0];
        firstUV[2][w][lane] = v2[0];
        __syncthreads();
        const int wb = min(w + 1, NW - 1);
        const float2 ub = firstUV[0][wb][lane], v1b = firstUV[1][wb][lane], v2b = firstUV[2][wb][lane];
        if (q.edge)
            dual(std::true_type{}, ub, v1b, v2b);
        else
            dual(std::false_type{}, ub, v1b, v2b);
        lastPQ[0][w][lane] = p2[R - 1];
        lastPQ[1][w][lane] = q2[R - 1];
        lastPQ[2][w][lane] = q3[R - 1];
        __syncthreads();
        const int wa = max(w - 1, 0);
        const float2 p2u = top ? splat(0.f) : lastPQ[0][wa][lane], q2u = top ? splat(0.f) : lastPQ[1][wa][lane],
                     q3u = top ? splat(0.f) : lastPQ[2][wa][lane];
        if (q.edge)
            primal(std::true_type{}, p2u, q2u, q3u, sum);
        else
            primal(std::false_type{}, p2u, q2u, q3u, sum);
    });
#pragma unroll
    for (int r = 0; r < R; r++) {
        q.store(a.un, r, u[r]);
        if (a.sn[0]) {
            q.store(a.sn[0], r, v1[r]);
            q.store(a.sn[1], r, v2[r]);
            q.store(a.sn[2], r, p1[r]);
            q.store(a.sn[3], r, p2[r]);
            q.store(a.sn[4], r, q1[r]);
            q.store(a.sn[5], r, q2[r]);
            q.store(a.sn[6], r, q3[r]);
        }
    }
    if (CHECK) store_partial(norms, fr.partials + tile_index<CHECK>(fr));
}

using Kernel = decltype(&k_tgv_strip2d<2, false>);
Kernel pick(int R, bool rule) {
    if (R == 2) return rule ? k_tgv_strip2d<2, true> : k_tgv_strip2d<2, false>;
    if (R == 3) return rule ? k_tgv_strip2d<3, true> : k_tgv_strip2d<3, false>;
    return rule ? k_tgv_strip2d<4, true> : k_tgv_strip2d<4, false>;
}

// just under alpha^2 (0 where that vanishes or alpha is not a positive number)
float near_square(float alpha) {
    const double v = (double)alpha * alpha * (1.0 - 1e-6);
    return v > 0.0 && alpha > 0.0f ? (float)std::min(v, (double)FLT_MAX) : 0.0f;
}

}  // namespace

bool tgv_strip_applies(const Dims& d) {
    const char* ek = getenv("CILREG_TGV_KERNEL");
    return strip::applies(d) && !(ek && ek[0] != '\0');
}

int tgv_strip_run(const float* f, float* u_out, float lam, float alpha1, float alpha0, int iters, float L2,
                  float epsil, const Dims& d, cudaStream_t s, float* info) {
    static const Choices choices = {1, 3, {2, 3, 4}, {1, 1, 1}, 400.0, 1230.0, 2000.0, 1770.0};
    const bool checking = epsil != 0.0f;
    const Plan P = plan(d.nx, d.ny, iters, checking, choices);
    Scratch scratch(s);
    IterControl ctl(s, scratch, iters, epsil, P.nblocks, 2);
    CILREG_TRY(ctl.status());
    const size_t bytes = sizeof(float) * (size_t)d.n;
    if (iters <= 0) CILREG_CUDA(cudaMemcpyAsync(u_out, f, bytes, cudaMemcpyDeviceToDevice, s));
    const int nl = count_spans(iters, P.T, checking);
    // launch k writes U to ub[(nl - 1 - k) & 1] (the last one u_out), the rest to set[k & 1]
    float *ub[2] = {u_out, nullptr}, *set[2][NS] = {};
    if (nl > 1) {
        ub[1] = scratch.floats(d.n);
        for (int i = 0; i < 2; i++)
            for (int c = 0; c < NS; c++) set[i][c] = scratch.floats(d.n);
    }
    if (scratch.status() != OK) return scratch.status();
    Args a = {};
    a.f = f;
    a.lambda = lam;
    a.alpha1 = alpha1;
    a.alpha0 = alpha0;
    a.near1 = near_square(alpha1);
    a.near0 = near_square(alpha0);
    a.tau = (float)pow((double)L2, -0.5);  // TGV_core.c:54-55
    a.inv_lt = 1.0f / (a.lambda + a.tau);
    CILREG_TRY(run_spans(P, ctl, iters, checking, d, host_aligned8(f) && host_aligned8(u_out),
                         [&](int k, const Span&, const Frame& fr) -> int {
                             a.u = k == 0 ? f : ub[(nl - k) & 1];
                             a.un = ub[(nl - 1 - k) & 1];
                             for (int c = 0; c < NS; c++) {
                                 a.s[c] = k == 0 ? nullptr : set[(k + 1) & 1][c];
                                 a.sn[c] = k == nl - 1 ? nullptr : set[k & 1][c];
                             }
                             CILREG_CUDA(launch_strip(pick(P.R, checking), P, fr, checking, s, a));
                             return OK;
                         }));
    if (checking && nl > 1) {
        const SpanResult r = span_result(ub, nl, u_out);
        CILREG_TRY(launch_take_span(ctl.ctl(), nl - 1, &r, 1, d.n, s));
    }
    return ctl.finish(info);
}

}  // namespace cilreg
