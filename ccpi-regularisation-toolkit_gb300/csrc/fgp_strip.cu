// FGP-TV and FGP-dTV on 2D images, several iterations per launch (strip2d.cuh),
// operation by operation with the arithmetic of the kernel that runs such images
// in a batch (FGP_TV_core.c:40-171, FGP_dTV_core.c:46-180): k_fgp_x2_2d's where
// the rows are even, k_fgp_stream's where they are odd, so that a batch of either
// equals its single calls bit for bit.  The two differ in which product of a sum
// of two is rounded (dot2).
//
// A thread holds P^{k-1}, P^{k-2} and f (and b) of its rows: R takes the place
// of P^{k-2} once it is formed, and P^{k-1} that of R once P^k is.  U of the
// row under a strip is recomputed from that row's R, which its warp publishes;
// U itself is never exchanged or stored but for the last iteration and the
// stopping checks.  The first launch of a cold run starts from zero duals
// without loading them, and no launch but a warm run's last stores the duals
// that nothing reads.
#include <vector>

#include "fgp_tiled.cuh"
#include "strip2d.cuh"

namespace cilreg {

namespace {

using namespace strip;

struct Args {
    const float* pc[2];  // P^{k-1}; null: zero
    const float* po[2];  // P^{k-2}
    float* qc[2];        // P of the launch's last iteration; null: not stored
    float* qo[2];        // P of the one before; null: not stored
    const float* f;
    const float* b[2];  // FGP-dTV: the reference's unit gradient
    float* u;           // output
    const float* u_prev;  // of a launch of one check iteration
    float lam, multip;
    float c[MAXT];  // momentum coefficients
    bool nonneg, aniso, write_u;
};

// a1 b1 + a2 b2
template <bool ODD>
__device__ __forceinline__ float2 dot2(float2 a1, float2 b1, float2 a2, float2 b2) {
    return ODD ? fma2(a1, b1, mul2(a2, b2)) : fma2(a2, b2, mul2(a1, b1));
}

// p scaled into the unit ball or clipped (utils.c:180-213)
template <bool ODD>
__device__ __forceinline__ void project(float2& p1, float2& p2, bool aniso) {
    if (!aniso) {
        const float2 den = dot2<ODD>(p1, p1, p2, p2);
        const float2 sq = make_float2((den.x > 1.f) ? rsqrt_normal(den.x) : 1.f,
                                      (den.y > 1.f) ? rsqrt_normal(den.y) : 1.f);
        p1 = mul2(p1, sq);
        p2 = mul2(p2, sq);
    } else {
        p1 = make_float2(unit_clip(p1.x), unit_clip(p1.y));
        p2 = make_float2(unit_clip(p2.x), unit_clip(p2.y));
    }
}

template <int R, bool CHECK, bool DTV, bool ODD>
__global__ void __launch_bounds__(NT, R <= 2 || (R == 3 && !DTV) ? 2 : 1)
    k_fgp_strip2d(Args a, Frame fr) {
    __shared__ float2 first1[2][NW][32], first2[2][NW][32], last2[2][NW][32];
    const Place<R> q(fr, CHECK, max(tile_index<CHECK>(fr), 0));
    const int lane = q.lane, w = q.w;
    // f and b never change during a run: loaded before the wait
    float2 f[R + 1], b1[DTV ? R : 1], b2[DTV ? R : 1];
#pragma unroll
    for (int r = 0; r <= R; r++) f[r] = q.load_const(a.f, r);
    if (DTV) {
#pragma unroll
        for (int r = 0; r < R; r++) {
            b1[r] = q.load_const(a.b[0], r);
            b2[r] = q.load_const(a.b[1], r);
        }
    }
    if (!begin<CHECK>(fr)) return;
    __shared__ float2 uo[CHECK ? R : 1][NW][32];  // U of the iteration before the check, each thread its own
    float2 p1[R], p2[R], o1[R], o2[R];  // o: P^{k-2}, then R
#pragma unroll
    for (int r = 0; r < R; r++) {
        p1[r] = a.pc[0] ? q.load(a.pc[0], r) : splat(0.f);
        p2[r] = a.pc[0] ? q.load(a.pc[1], r) : splat(0.f);
        o1[r] = a.pc[0] ? q.load(a.po[0], r) : splat(0.f);
        o2[r] = a.pc[0] ? q.load(a.po[1], r) : splat(0.f);
        if (CHECK && fr.count == 1) uo[CHECK ? r : 0][w][lane] = q.load(a.u_prev, r);
    }
    const float2 mlam2 = splat(-a.lam), mp2 = splat(a.multip);
    const bool top = q.Y == 0;
    Norms norms;

    auto iterate = [&](auto edge_, float2 r2up, float2 r1dn, float2 r2dn, int t, auto last) {
        constexpr bool EDGE = decltype(edge_)::value;
        // U = f - lambda div R, zero flux below index 0 (FGP_TV_core.c:220-236)
        auto u_of = [&](float2 r1, float2 r2, float2 r2above, float2 fv) -> float2 {
            float lo = left_of(r1);
            if (EDGE && q.at_left) lo = 0.f;
            const float2 s = sub2(sub2(add2(r1, r2), make_float2(lo, r1.x)), r2above);
            float2 u = fma2(mlam2, s, fv);
            if (a.nonneg) u = make_float2(u.x < 0.f ? 0.f : u.x, u.y < 0.f ? 0.f : u.y);
            return u;
        };
        float2 u = u_of(o1[0], o2[0], r2up, f[0]);
#pragma unroll
        for (int r = 0; r < R; r++) {
            constexpr int N = R - 1;
            const float2 un = r < N ? u_of(o1[r < N ? r + 1 : 0], o2[r < N ? r + 1 : 0], o2[r], f[r + 1])
                                    : u_of(r1dn, r2dn, o2[r], f[R]);
            const float hi = right_of(u);
            float2 g1 = make_float2(u.x - u.y, u.y - hi);
            float2 g2 = sub2(u, un);
            if (EDGE) {
                if (q.odd_end) g1.x = 0.f;
                if (q.at_right) g1.y = 0.f;
                if (r == q.bottom) g2 = splat(0.f);
            }
            if (DTV) {
                const float2 c1 = b1[DTV ? r : 0], c2 = b2[DTV ? r : 0];
                const float2 ip = dot2<ODD>(g1, c1, g2, c2);
                g1 = fma2(neg2(ip), c1, g1);
                g2 = fma2(neg2(ip), c2, g2);
            }
            float2 n1 = fma2(mp2, g1, o1[r]), n2 = fma2(mp2, g2, o2[r]);
            project<ODD>(n1, n2, a.aniso);
            if (last && a.write_u) {
                if (CHECK) add_norms(q, r, u, uo[CHECK ? r : 0][w][lane], norms);
                q.store(a.u, r, u);
            }
            if (CHECK && t == fr.count - 2) uo[CHECK ? r : 0][w][lane] = u;
            o1[r] = p1[r];
            o2[r] = p2[r];
            p1[r] = n1;
            p2[r] = n2;
            u = un;
        }
    };
    iterations<CHECK>(fr.count, [&](int t, auto last) {
        const float2 cm = splat(a.c[t]);
#pragma unroll
        for (int r = 0; r < R; r++) {
            float2 r1 = fma2(cm, sub2(p1[r], o1[r]), p1[r]), r2 = fma2(cm, sub2(p2[r], o2[r]), p2[r]);
            if (DTV) {
                const float2 c1 = b1[DTV ? r : 0], c2 = b2[DTV ? r : 0];
                const float2 ip = dot2<ODD>(r1, c1, r2, c2);
                r1 = fma2(neg2(ip), c1, r1);
                r2 = fma2(neg2(ip), c2, r2);
            }
            o1[r] = r1;
            o2[r] = r2;
        }
        const int s = t & 1;
        first1[s][w][lane] = o1[0];
        first2[s][w][lane] = o2[0];
        last2[s][w][lane] = o2[R - 1];
        __syncthreads();
        const float2 r2up = top ? splat(0.f) : (w > 0 ? last2[s][w - 1][lane] : o2[0]);
        const float2 r1dn = w < NW - 1 ? first1[s][w + 1][lane] : o1[R - 1];
        const float2 r2dn = w < NW - 1 ? first2[s][w + 1][lane] : o2[R - 1];
        if (q.edge)
            iterate(std::true_type{}, r2up, r1dn, r2dn, t, last);
        else
            iterate(std::false_type{}, r2up, r1dn, r2dn, t, last);
    });
#pragma unroll
    for (int r = 0; r < R; r++) {
        if (a.qc[0]) {
            q.store(a.qc[0], r, p1[r]);
            q.store(a.qc[1], r, p2[r]);
        }
        if (a.qo[0]) {
            q.store(a.qo[0], r, o1[r]);
            q.store(a.qo[1], r, o2[r]);
        }
    }
    if (CHECK) store_partial(norms, fr.partials + tile_index<CHECK>(fr));
}

using Kernel = decltype(&k_fgp_strip2d<2, false, false, false>);
template <bool DTV, bool ODD>
Kernel pick_r(int R, bool check) {
    if (R == 2) return check ? k_fgp_strip2d<2, true, DTV, ODD> : k_fgp_strip2d<2, false, DTV, ODD>;
    if (R == 3) return check ? k_fgp_strip2d<3, true, DTV, ODD> : k_fgp_strip2d<3, false, DTV, ODD>;
    return check ? k_fgp_strip2d<4, true, DTV, ODD> : k_fgp_strip2d<4, false, DTV, ODD>;
}
Kernel pick(int R, bool check, bool dtv, bool odd) {
    if (odd) return dtv ? pick_r<true, true>(R, check) : pick_r<false, true>(R, check);
    return dtv ? pick_r<true, false>(R, check) : pick_r<false, false>(R, check);
}

}  // namespace

bool fgp_strip_applies(const Dims& d) {
    const char* ek = getenv("CILREG_FGP_KERNEL");
    return strip::applies(d) && !(ek && ek[0] != '\0');
}

int fgp_strip_run(const float* f, const float* const* b, float* u_out, float lam, float multip,
                  const std::vector<float>& cseq, float epsil, bool nonneg, bool aniso, const Dims& d, cudaStream_t s,
                  float* info, FgpWarm* warm) {
    static const Choices tv = {1, 3, {2, 3, 4}, {2, 2, 1}, 840.0, 310.0, 1200.0, 1150.0};
    static const Choices dtv = {1, 3, {2, 3, 4}, {2, 1, 1}, 860.0, 340.0, 1200.0, 1200.0};
    const int iters = (int)cseq.size();
    const bool checking = epsil != 0.0f;
    const Plan P = plan(d.nx, d.ny, iters, checking, b ? dtv : tv);
    Scratch scratch(s);
    IterControl ctl(s, scratch, iters, epsil, P.nblocks, 2);
    CILREG_TRY(ctl.status());
    const int nl = count_spans(iters, P.T, checking);
    // launch k writes (P, P before) to set[k & 1] and reads set[(k + 1) & 1]
    float* set[2][4] = {};
    for (int i = 0; i < 2; i++)
        for (int c = 0; c < 4; c++)
            if (nl > 1 || (warm && checking)) {
                set[i][c] = scratch.floats(d.n);
                if (!set[i][c]) return scratch.status();
            }
    Args a = {};
    a.f = f;
    a.u_prev = u_out;
    a.lam = lam;
    a.multip = multip;
    a.nonneg = nonneg;
    a.aniso = aniso;
    bool aligned = host_aligned8(f) && host_aligned8(u_out);
    for (int c = 0; c < 2 && b; c++) {
        a.b[c] = b[c];
        aligned = aligned && host_aligned8(b[c]);
    }
    // a warm run starts from the newest duals of the caller's ring and leaves
    // its own in the buffer after it; its first coefficient is 0, so the
    // duals before the newest never count
    const int from = warm ? (warm->base + 2) % 3 : 0, to = warm ? warm->base : 0;
    // U of a check must outlive the launch that carries the check: two buffers,
    // of which the last launch writes u_out
    float* ualt = checking && nl > 1 ? scratch.floats(d.n) : nullptr;
    if (checking && nl > 1 && !ualt) return scratch.status();
    CILREG_TRY(run_spans(P, ctl, iters, checking, d, aligned, [&](int k, const Span& sp, const Frame& fr) -> int {
        const bool end = k == nl - 1;
        for (int c = 0; c < 2; c++) {
            a.pc[c] = k > 0 ? set[(k + 1) & 1][c] : warm ? warm->ring[from][c] : nullptr;
            a.po[c] = k > 0 ? set[(k + 1) & 1][2 + c] : a.pc[c];
            a.qc[c] = set[k & 1][c];
            a.qo[c] = set[k & 1][2 + c];
            if (end && !(warm && checking)) {
                a.qc[c] = warm ? warm->ring[to][c] : nullptr;
                a.qo[c] = nullptr;
            }
        }
        for (int t = 0; t < sp.count; t++) a.c[t] = cseq[sp.first + t];
        a.u = (checking && ((nl - 1 - k) & 1)) ? ualt : u_out;
        a.write_u = end || sp.check;
        CILREG_CUDA(launch_strip(pick(P.R, checking, b != nullptr, d.nx & 1), P, fr, checking, s, a));
        return OK;
    }));
    // what the check that fired, or the last launch, left: U, and a warm run's duals
    SpanResult r[3];
    int nr = 0;
    if (checking && nl > 1) {
        float* const ub[2] = {u_out, ualt};
        r[nr++] = span_result(ub, nl, u_out);
    }
    for (int c = 0; c < 2 && warm && checking && iters > 0; c++)
        r[nr++] = SpanResult{{set[0][c], set[1][c]}, warm->ring[to][c], false};
    if (nr > 0) CILREG_TRY(launch_take_span(ctl.ctl(), nl - 1, r, nr, d.n, s));
    CILREG_TRY(ctl.finish(info));
    if (warm && iters > 0) warm->base = (to + 1) % 3;
    return OK;
}

}  // namespace cilreg
