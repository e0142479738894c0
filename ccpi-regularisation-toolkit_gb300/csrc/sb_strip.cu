// Split-Bregman TV on 2D images, several outer iterations per launch
// (strip2d.cuh).  As in k_sb_fused, the state is (U^k, B^{k-1}): an iteration
// forms D^k, B^k from it and runs both Jacobi sweeps (SB_TV_core.c:149-371).
// The shrinkage of the row above a strip is recomputed from that row's U and
// B; the first sweep's U1 is exchanged after a second barrier.
#include "sb_tiled.cuh"
#include "strip2d.cuh"

namespace cilreg {

namespace {

using namespace strip;

struct Args {
    const float* u;      // U^k
    float* un;           // U after the launch
    const float* bp[2];  // B^{k-1}; of the first iteration: B^0, null for zero
    const float* d0[2];  // of the first iteration: D^0, null for zero
    float* bn[2];        // B after the launch; null: not stored
    const float* f;
    float lambda, mu, norm, dlam;
    bool first;  // the launch starts with iteration 0, whose D and B are given
    bool aniso;
};

// D - B and B of a pair after a shrinkage
__device__ __forceinline__ void shrink(float2 g1, float2 g2, float2 b1, float2 b2, float dlam, bool aniso, float2& q1,
                                       float2& q2, float2& n1, float2& n2) {
    const float2 g[2] = {g1, g2}, b[2] = {b1, b2};
    float2 d[2], n[2];
    sb_shrink2(g, b, dlam, aniso, d, n);
    n1 = n[0];
    n2 = n[1];
    q1 = sub2(d[0], n[0]);
    q2 = sub2(d[1], n[1]);
}

template <int R, bool CHECK>
__global__ void __launch_bounds__(NT, R <= 2 ? 2 : 1) k_sb_strip2d(Args a, Frame fr) {
    __shared__ float2 firstU[NW][32], lastU[NW][32], lastB1[NW][32], lastB2[NW][32], first1[NW][32], last1[NW][32];
    const Place<R> q(fr, CHECK, max(tile_index<CHECK>(fr), 0));
    const int lane = q.lane, w = q.w;
    float2 muf[R], u[R], b1[R], b2[R];
#pragma unroll
    for (int r = 0; r < R; r++) muf[r] = mul2(splat(a.mu), q.load_const(a.f, r));  // before the wait
    if (!begin<CHECK>(fr)) return;
    const bool top = q.Y == 0;
    float2 q1[R], q2[R], q2up = splat(0.f);  // D - B
#pragma unroll
    for (int r = 0; r < R; r++) {
        u[r] = q.load(a.u, r);
        b1[r] = a.bp[0] ? q.load(a.bp[0], r) : splat(0.f);
        b2[r] = a.bp[0] ? q.load(a.bp[1], r) : splat(0.f);
        q1[r] = q2[r] = splat(0.f);
    }
    if (a.first && a.d0[0]) {  // given D^0, B^0: of the rows and of the one above
#pragma unroll
        for (int r = 0; r < R; r++) {
            q1[r] = sub2(q.load(a.d0[0], r), b1[r]);
            q2[r] = sub2(q.load(a.d0[1], r), b2[r]);
        }
        const int up = top ? 1 : -1;  // row -1 of the image is the mirrored row 1
        q2up = sub2(q.load(a.d0[1], up), q.load(a.bp[1], up));
    }
    const float2 lam2 = splat(a.lambda), norm2 = splat(a.norm);
    Norms norms;
    float2 g[R], u1[R];

    auto sum4 = [](float2 xh, float2 xl, float2 yh, float2 yl) { return add2(add2(add2(xh, xl), yh), yl); };
    // D, B, their divergence term G and the first sweep
    auto sweep1 = [&](auto edge_, float2 above, float2 next, float2 below, float2 b1a, float2 b2a, bool given) {
        constexpr bool EDGE = decltype(edge_)::value;
        if (!given) {  // the row above: its y component
            float2 c = above, e1, n1, n2;
            float lo, hi;
            x_neighbours<EDGE>(q, c, lo, hi);
            shrink(sub2(make_float2(c.y, hi), c), sub2(next, c), b1a, b2a, a.dlam, a.aniso, e1, q2up, n1, n2);
        }
        float2 um = above, ql = q2up;
#pragma unroll
        for (int r = 0; r < R; r++) {
            float2 c = u[r];
            float lo, hi;
            x_neighbours<EDGE>(q, c, lo, hi);
            const float2 xl = make_float2(lo, c.x), xh = make_float2(c.y, hi);
            float2 uh = (r < R - 1) ? u[r + 1 < R ? r + 1 : r] : below;
            if (EDGE && r == q.bottom) uh = um;
            if (!given) {
                float2 n1, n2;
                shrink(sub2(xh, c), sub2(uh, c), b1[r], b2[r], a.dlam, a.aniso, q1[r], q2[r], n1, n2);
                b1[r] = n1;
                b2[r] = n2;
            }
            float qxl = left_of(q1[r]);
            if (EDGE && q.at_left) qxl = q1[r].y;
            // Dx[-1] - Dx + Dy[-1] - Dy - Bx[-1] + Bx - By[-1] + By (SB_TV_core.c:166)
            float2 s = sub2(make_float2(qxl, q1[r].x), q1[r]);
            s = sub2(add2(s, ql), q2[r]);
            g[r] = s;
            u1[r] = mul2(norm2, fma2(add2(s, sum4(xh, xl, uh, um)), lam2, muf[r]));
            um = u[r];
            ql = q2[r];
        }
    };
    auto sweep2 = [&](auto edge_, float2 above, float2 below, auto sum) {
        constexpr bool EDGE = decltype(edge_)::value;
        float2 um = above;
#pragma unroll
        for (int r = 0; r < R; r++) {
            float2 c = u1[r];
            float lo, hi;
            x_neighbours<EDGE>(q, c, lo, hi);
            float2 uh = (r < R - 1) ? u1[r + 1 < R ? r + 1 : r] : below;
            if (EDGE && r == q.bottom) uh = um;
            const float2 s = add2(g[r], sum4(make_float2(c.y, hi), make_float2(lo, c.x), uh, um));
            const float2 un = mul2(norm2, fma2(s, lam2, muf[r]));
            if (CHECK && sum) add_norms(q, r, un, u1[r], norms);
            u[r] = un;
            um = u1[r];
        }
    };
    iterations<CHECK>(fr.count, [&](int t, auto sum) {
        firstU[w][lane] = u[0];
        lastU[w][lane] = u[R - 1];
        lastB1[w][lane] = b1[R - 1];
        lastB2[w][lane] = b2[R - 1];
        __syncthreads();
        const float2 below = w < NW - 1 ? firstU[w + 1][lane] : u[R - 1];
        const float2 above = top ? u[1] : (w > 0 ? lastU[w - 1][lane] : u[0]);
        const float2 next = top ? (q.ny == 2 ? u[0] : (R > 2 ? u[R > 2 ? 2 : 0] : below)) : u[0];
        const float2 b1a = top ? b1[1] : (w > 0 ? lastB1[w - 1][lane] : b1[0]);
        const float2 b2a = top ? b2[1] : (w > 0 ? lastB2[w - 1][lane] : b2[0]);
        const bool given = a.first && t == 0;
        if (q.edge)
            sweep1(std::true_type{}, above, next, below, b1a, b2a, given);
        else
            sweep1(std::false_type{}, above, next, below, b1a, b2a, given);
        first1[w][lane] = u1[0];
        last1[w][lane] = u1[R - 1];
        __syncthreads();
        const float2 below1 = w < NW - 1 ? first1[w + 1][lane] : u1[R - 1];
        const float2 above1 = top ? u1[1] : (w > 0 ? last1[w - 1][lane] : u1[0]);
        if (q.edge)
            sweep2(std::true_type{}, above1, below1, sum);
        else
            sweep2(std::false_type{}, above1, below1, sum);
    });
#pragma unroll
    for (int r = 0; r < R; r++) {
        q.store(a.un, r, u[r]);
        if (a.bn[0]) {
            q.store(a.bn[0], r, b1[r]);
            q.store(a.bn[1], r, b2[r]);
        }
    }
    if (CHECK) store_partial(norms, fr.partials + tile_index<CHECK>(fr));
}

using Kernel = decltype(&k_sb_strip2d<2, false>);
Kernel pick(int R, bool rule) {
    if (R == 2) return rule ? k_sb_strip2d<2, true> : k_sb_strip2d<2, false>;
    if (R == 3) return rule ? k_sb_strip2d<3, true> : k_sb_strip2d<3, false>;
    return rule ? k_sb_strip2d<4, true> : k_sb_strip2d<4, false>;
}

}  // namespace

bool sb_strip_applies(const Dims& d) {
    const char* ek = getenv("CILREG_SB_KERNEL");
    return strip::applies(d) && !(ek && ek[0] != '\0');
}

int sb_strip_run(const SbSweepArgs& in, float dlam, bool aniso, float* u_out, int iters, float epsil, const Dims& d,
                 cudaStream_t s, float* info, SbWarm* warm) {
    static const Choices choices = {2, 3, {2, 3, 4}, {2, 1, 1}, 910.0, 430.0, 870.0, 1070.0};
    const bool checking = epsil != 0.0f;
    const Plan P = plan(d.nx, d.ny, iters, checking, choices);
    Scratch scratch(s);
    IterControl ctl(s, scratch, iters, epsil, P.nblocks, 2);
    CILREG_TRY(ctl.status());
    const size_t bytes = sizeof(float) * (size_t)d.n;
    if (iters <= 0) CILREG_CUDA(cudaMemcpyAsync(u_out, in.f, bytes, cudaMemcpyDeviceToDevice, s));
    const int nl = count_spans(iters, P.T, checking);
    // launch k writes U to ub[(nl - 1 - k) & 1] (the last one u_out), B to bb[k & 1]
    float *ub[2] = {u_out, nullptr}, *bb[2][2] = {};
    if (nl > 1) ub[1] = scratch.floats(d.n);
    for (int i = 0; i < 2 && (nl > 1 || warm); i++)
        for (int c = 0; c < 2; c++) bb[i][c] = scratch.floats(d.n);
    if (scratch.status() != OK) return scratch.status();
    Args a = {};
    a.f = in.f;
    a.lambda = in.lambda;
    a.mu = in.mu;
    a.norm = in.norm;
    a.dlam = dlam;
    a.aniso = aniso;
    CILREG_TRY(run_spans(P, ctl, iters, checking, d, host_aligned8(in.f) && host_aligned8(u_out),
                         [&](int k, const Span&, const Frame& fr) -> int {
                             a.first = k == 0;
                             a.u = k == 0 ? in.f : ub[(nl - k) & 1];
                             a.un = ub[(nl - 1 - k) & 1];
                             for (int c = 0; c < 2; c++) {
                                 a.d0[c] = warm ? warm->dd[c] : nullptr;
                                 a.bp[c] = k > 0 ? bb[(k + 1) & 1][c] : warm ? warm->bb[c] : nullptr;
                                 a.bn[c] = (k == nl - 1 && !warm) ? nullptr : bb[k & 1][c];
                             }
                             CILREG_CUDA(launch_strip(pick(P.R, checking), P, fr, checking, s, a));
                             return OK;
                         }));
    // what the check that fired, or the last launch, left: U, and a warm run's B of
    // the iteration before, from which it shrinks once more with that U
    SpanResult r[3];
    int nr = 0;
    if (checking && nl > 1) r[nr++] = span_result(ub, nl, u_out);
    for (int c = 0; c < 2 && warm && iters > 0; c++) r[nr++] = SpanResult{{bb[0][c], bb[1][c]}, warm->bb[c], false};
    if (nr > 0) CILREG_TRY(launch_take_span(ctl.ctl(), nl - 1, r, nr, d.n, s));
    if (warm && iters > 0) {
        StopCtl* never = (StopCtl*)scratch.bytes(sizeof(StopCtl));
        if (!never) return scratch.status();
        CILREG_CUDA(cudaMemsetAsync(never, 0, sizeof(StopCtl), s));
        CILREG_TRY(sb_shrink2d(in, dlam, aniso, u_out, *warm, d, never, s));
    }
    return ctl.finish(info);
}

}  // namespace cilreg
