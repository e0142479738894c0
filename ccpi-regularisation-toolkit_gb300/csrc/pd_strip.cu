// PD-TV on 2D images, several iterations per launch (strip2d.cuh), with the
// reference's rounding of every operation (pd_math.cuh, PD_TV_core.c:40-252)
// and so k_pd_2d's bits.  Additions and subtractions issue paired; products
// that feed one stay scalar (mul2_rn).  The projected dual of the row above a
// strip is exchanged after a second barrier: its square root and division
// cost more than the barrier.
#include "pd_math.cuh"
#include "pd_tiled.cuh"
#include "strip2d.cuh"

namespace cilreg {

namespace {

using namespace strip;

struct Args {
    const float* u;     // extrapolated iterate; P^0 = 0 where p is null
    const float* p[2];
    float* un;          // extrapolated iterate after the launch
    float* pn[2];       // null: not stored
    float* brk;         // U before the extrapolation, of a check
    const float* f;
    float sigma, tau, lt;
    DoubleDivisor onelt;
    bool nonneg, aniso;
};

template <int R, bool CHECK>
__global__ void __launch_bounds__(NT, R <= 3 ? 2 : 1) k_pd_strip2d(Args a, Frame fr) {
    __shared__ float2 firstU[NW][32], lastU[NW][32], lastP[NW][32];
    const Place<R> q(fr, CHECK, max(tile_index<CHECK>(fr), 0));
    const int lane = q.lane, w = q.w;
    float2 ltf[R], u[R], p1[R], p2[R];
#pragma unroll
    for (int r = 0; r < R; r++) ltf[r] = mul2_rn(splat(a.lt), q.load_const(a.f, r));  // before the wait
    if (!begin<CHECK>(fr)) return;
#pragma unroll
    for (int r = 0; r < R; r++) {
        u[r] = q.load(a.u, r);
        p1[r] = a.p[0] ? q.load(a.p[0], r) : splat(0.f);
        p2[r] = a.p[0] ? q.load(a.p[1], r) : splat(0.f);
    }
    const float2 sigma2 = splat(a.sigma), tau2 = splat(a.tau);
    Norms norms;

    // P += sigma grad U, projected (mirrored differences at the far edges)
    auto dual = [&](auto edge_, float2 above, float2 below) {
        constexpr bool EDGE = decltype(edge_)::value;
        float2 um = above;
#pragma unroll
        for (int r = 0; r < R; r++) {
            float2 c = u[r];
            float hi = right_of(c);
            if (EDGE) {
                const float lo = left_of(c);
                if (q.odd_end) c.y = lo;
                if (q.at_right) hi = c.x;
            }
            float2 uh = (r < R - 1) ? u[r + 1 < R ? r + 1 : r] : below;
            if (EDGE && r == q.bottom) uh = um;
            float2 n1 = add2(p1[r], mul2_rn(sigma2, sub2(make_float2(c.y, hi), c)));
            float2 n2 = add2(p2[r], mul2_rn(sigma2, sub2(uh, c)));
            if (!a.aniso) {
                const float2 den = add2(mul2_rn(n1, n1), mul2_rn(n2, n2));
                if (den.x > 1.0f) {
                    const float s = __fdiv_rn(1.0f, __fsqrt_rn(den.x));
                    n1.x = __fmul_rn(n1.x, s);
                    n2.x = __fmul_rn(n2.x, s);
                }
                if (den.y > 1.0f) {
                    const float s = __fdiv_rn(1.0f, __fsqrt_rn(den.y));
                    n1.y = __fmul_rn(n1.y, s);
                    n2.y = __fmul_rn(n2.y, s);
                }
            } else {
                n1 = make_float2(unit_clip(n1.x), unit_clip(n1.y));
                n2 = make_float2(unit_clip(n2.x), unit_clip(n2.y));
            }
            p1[r] = n1;
            p2[r] = n2;
            um = u[r];
        }
    };
    auto primal = [&](auto edge_, float2 p2up, auto sum) {
        constexpr bool EDGE = decltype(edge_)::value;
#pragma unroll
        for (int r = 0; r < R; r++) {
            float lo = left_of(p1[r]);
            if (EDGE && q.at_left) lo = 0.f;
            // div = -(P1 - P1[-1]) - (P2 - P2[-1]), P[-1] = 0
            const float2 dv = add2(sub2(make_float2(lo, p1[r].x), p1[r]), sub2(p2up, p2[r]));
            float2 uc = u[r];
            if (a.nonneg) uc = make_float2(uc.x < 0.f ? 0.f : uc.x, uc.y < 0.f ? 0.f : uc.y);
            const float2 un = div_by_double2(add2(sub2(uc, mul2_rn(tau2, dv)), ltf[r]), a.onelt);
            if (CHECK && sum) {
                add_norms(q, r, un, uc, norms);
                q.store(a.brk, r, un);
            }
            u[r] = add2(un, sub2(un, uc));  // theta = 1
            p2up = p2[r];
        }
    };
    iterations<CHECK>(fr.count, [&](int t, auto sum) {
        firstU[w][lane] = u[0];
        lastU[w][lane] = u[R - 1];
        __syncthreads();
        const float2 below = w < NW - 1 ? firstU[w + 1][lane] : u[R - 1];
        const float2 above = w > 0 ? lastU[w - 1][lane] : u[0];
        if (q.edge)
            dual(std::true_type{}, above, below);
        else
            dual(std::false_type{}, above, below);
        lastP[w][lane] = p2[R - 1];
        __syncthreads();
        const float2 p2up = q.Y == 0 ? splat(0.f) : (w > 0 ? lastP[w - 1][lane] : p2[0]);
        if (q.edge)
            primal(std::true_type{}, p2up, sum);
        else
            primal(std::false_type{}, p2up, sum);
    });
#pragma unroll
    for (int r = 0; r < R; r++) {
        q.store(a.un, r, u[r]);
        if (a.pn[0]) {
            q.store(a.pn[0], r, p1[r]);
            q.store(a.pn[1], r, p2[r]);
        }
    }
    if (CHECK) store_partial(norms, fr.partials + tile_index<CHECK>(fr));
}

using Kernel = decltype(&k_pd_strip2d<2, false>);
Kernel pick(int R, bool rule) {
    if (R == 2) return rule ? k_pd_strip2d<2, true> : k_pd_strip2d<2, false>;
    if (R == 3) return rule ? k_pd_strip2d<3, true> : k_pd_strip2d<3, false>;
    return rule ? k_pd_strip2d<4, true> : k_pd_strip2d<4, false>;
}

}  // namespace

bool pd_strip_applies(const Dims& d) {
    const char* ek = getenv("CILREG_PD_KERNEL");
    return strip::applies(d) && !(ek && ek[0] != '\0');
}

int pd_strip_run(const float* f, float* u_out, float sigma, float tau, float lt, const DoubleDivisor& onelt, int iters,
                 float epsil, bool nonneg, bool aniso, const Dims& d, cudaStream_t s, float* info) {
    static const Choices choices = {1, 3, {2, 3, 4}, {2, 2, 1}, 560.0, 665.0, 1250.0, 750.0};
    const bool checking = epsil != 0.0f;
    const Plan P = plan(d.nx, d.ny, iters, checking, choices);
    Scratch scratch(s);
    IterControl ctl(s, scratch, iters, epsil, P.nblocks, 2);
    CILREG_TRY(ctl.status());
    const size_t bytes = sizeof(float) * (size_t)d.n;
    if (iters <= 0) CILREG_CUDA(cudaMemcpyAsync(u_out, f, bytes, cudaMemcpyDeviceToDevice, s));
    const int nl = count_spans(iters, P.T, checking);
    // launch k writes U to ub[(nl - 1 - k) & 1] (the last one u_out) and P to
    // pb[k & 1]; a check also its U before the extrapolation to brk[k & 1],
    // which must outlive the launch that carries the check
    float *ub[2] = {u_out, nullptr}, *pb[2][2] = {}, *brk[2] = {};
    if (nl > 1) {
        ub[1] = scratch.floats(d.n);
        for (int i = 0; i < 2; i++)
            for (int c = 0; c < 2; c++) pb[i][c] = scratch.floats(d.n);
    }
    for (int i = 0; i < 2 && checking; i++) brk[i] = scratch.floats(d.n);
    if (scratch.status() != OK) return scratch.status();
    Args a = {};
    a.f = f;
    a.sigma = sigma;
    a.tau = tau;
    a.lt = lt;
    a.onelt = onelt;
    a.nonneg = nonneg;
    a.aniso = aniso;
    CILREG_TRY(run_spans(P, ctl, iters, checking, d, host_aligned8(f) && host_aligned8(u_out),
                         [&](int k, const Span&, const Frame& fr) -> int {
                             a.u = k == 0 ? f : ub[(nl - k) & 1];
                             a.un = ub[(nl - 1 - k) & 1];
                             a.brk = brk[k & 1];
                             for (int c = 0; c < 2; c++) {
                                 a.p[c] = k == 0 ? nullptr : pb[(k + 1) & 1][c];
                                 a.pn[c] = k == nl - 1 ? nullptr : pb[k & 1][c];
                             }
                             CILREG_CUDA(launch_strip(pick(P.R, checking), P, fr, checking, s, a));
                             return OK;
                         }));
    if (checking && iters > 0) {
        const SpanResult r = {{brk[0], brk[1]}, u_out, true};
        CILREG_TRY(launch_take_span(ctl.ctl(), nl - 1, &r, 1, d.n, s));
    }
    return ctl.finish(info);
}

}  // namespace cilreg
