// LLT-ROF on 2D images, several iterations per launch (strip2d.cuh), with the
// arithmetic of k_llt_pair2d (LLT_ROF_core.c:54-436).  A row's terms (the ROF
// fluxes R1, R2 and the second differences' signs L1, L2) are formed one row
// ahead of the row that is updated; the terms of the rows right above and
// below a strip, R1 and L2, are recomputed from the two rows on either side
// that the neighbouring warps publish, which costs less than exchanging them
// after a second barrier.
#include "llt.cuh"
#include "strip2d.cuh"

namespace cilreg {

namespace {

using namespace strip;

template <int R, bool CHECK>
__global__ void __launch_bounds__(NT, R <= 2 ? 2 : 1)
    k_llt_strip2d(const float* __restrict__ U, float* __restrict__ Un, const float* __restrict__ F, float lam_rof,
                  float lam_llt, float tau, Frame fr) {
    __shared__ float2 first[2][2][NW][32], last[2][2][NW][32];  // [slot][row from the end]
    const Place<R> q(fr, CHECK, max(tile_index<CHECK>(fr), 0));
    const int lane = q.lane, w = q.w;
    const bool odd = q.nx & 1;
    const float2 EPS2 = splat(1.0e-12f), MTWO2 = splat(-2.0f);
    const float2 tau2 = splat(tau), lrof2 = splat(lam_rof), mlllt2 = splat(-lam_llt);
    float2 f[R], u[R];
#pragma unroll
    for (int r = 0; r < R; r++) f[r] = q.load_const(F, r);  // never changes: loaded before the wait
    if (!begin<CHECK>(fr)) return;
#pragma unroll
    for (int r = 0; r < R; r++) u[r] = q.load(U, r);
    Norms norms;

    auto sign_terms = [](float2 v1, float2 v2, float2& t1, float2& t2) {
        t1 = llt_sign2(v1);
        t2 = llt_sign2(v2);
        if (llt_divides2(v1) | llt_divides2(v2)) {
            t1 = llt_quot2(v1);
            t2 = llt_quot2(v2);
        }
    };
    // row -1 is the mirrored row 1 at the image's first row: `above`, with its
    // own upper and lower rows above_h and above_l; below2 is the row under
    // the row under the strip
    auto iterate = [&](auto edge_, float2 above_l, float2 above, float2 above_h, float2 below, float2 below2, auto sum) {
        constexpr bool EDGE = decltype(edge_)::value;
        float2 r1l, l2l;  // R1 and L2 of the row above
        {
            float2 c = above;
            float lo, hi;
            x_neighbours<EDGE>(q, c, lo, hi);
            const float2 yp = sub2(above_h, c);
            const float2 mx2 = minmod_sq2(sub2(make_float2(c.y, hi), c), sub2(c, make_float2(lo, c.x)));
            r1l = normalise2(yp, add2(fma2(yp, yp, mx2), EPS2));
            const float2 v2 = add2(fma2(MTWO2, c, above_h), above_l);
            float2 unused;
            sign_terms(v2, v2, unused, l2l);
        }
        float2 r1, dv2, l2, dxx;  // of the row that is updated next
        float2 um = above;
#pragma unroll
        for (int r = 0; r <= R; r++) {
            // terms of row r (of the row under the strip, L2 only)
            float2 c = r < R ? u[r < R ? r : 0] : below;
            float2 uh = r < R - 1 ? u[r + 1 < R ? r + 1 : 0] : (r == R - 1 ? below : below2);
            if (EDGE && r == q.bottom) uh = um;  // mirrored: the row above is also the row below
            float2 n1 = splat(0.f), nv2 = splat(0.f), nl2, nxx = splat(0.f);
            const float2 v2 = add2(fma2(MTWO2, c, uh), um);
            if (r < R) {
                float lo, hi;
                x_neighbours<EDGE>(q, c, lo, hi);
                const float2 cl = make_float2(lo, c.x), ch = make_float2(c.y, hi);
                const float2 xp = sub2(ch, c), xm = sub2(c, cl);
                const float2 yp = sub2(uh, c), ym = sub2(c, um);
                const float2 mx2 = minmod_sq2(xp, xm), my2 = minmod_sq2(yp, ym);
                n1 = normalise2(yp, add2(fma2(yp, yp, mx2), EPS2));
                const float2 r2 = normalise2(xp, add2(fma2(xp, xp, my2), EPS2));
                float2 l1;
                sign_terms(add2(fma2(MTWO2, c, ch), cl), v2, l1, nl2);
                float llo, lhi, r2l = left_of(r2);
                x_neighbours<EDGE>(q, l1, llo, lhi);
                if (EDGE && q.at_left) r2l = r2.y;
                nv2 = sub2(r2, make_float2(r2l, r2.x));
                nxx = add2(fma2(MTWO2, l1, make_float2(l1.y, lhi)), make_float2(llo, l1.x));
            } else {
                float2 unused;
                sign_terms(v2, v2, unused, nl2);
            }
            if (r > 0) {  // update row r - 1
                const int k = r > 0 ? r - 1 : 0;
                const float2 l2h = (EDGE && k == q.bottom) ? l2l : nl2;
                const float2 dyy = add2(fma2(MTWO2, l2, l2h), l2l);
                const float2 dv1 = sub2(r1, r1l);
                const float2 lap = add2(dxx, dyy), div = add2(dv1, dv2);
                // odd rows round as the one-voxel kernel: the sign terms turn a
                // last-place difference into 5e-5 of the image in 1000 iterations
                const float2 g = odd ? fma2(lrof2, div, mul2(mlllt2, lap)) : fma2(mlllt2, lap, mul2(lrof2, div));
                const float2 t = sub2(g, sub2(um, f[k]));
                const float2 un = fma2(tau2, t, um);
                if (CHECK && sum) add_norms(q, k, un, um, norms);
                u[k] = un;
                r1l = r1;
                l2l = l2;
            }
            r1 = n1;
            dv2 = nv2;
            l2 = nl2;
            dxx = nxx;
            um = c;
        }
    };
    iterations<CHECK>(fr.count, [&](int t, auto sum) {
        const int b = t & 1;
        first[b][0][w][lane] = u[0];
        first[b][1][w][lane] = u[1];
        last[b][0][w][lane] = u[R - 1];
        last[b][1][w][lane] = u[R - 2];
        __syncthreads();
        const bool top = q.Y == 0, lowest = w == NW - 1;
        const float2 below = lowest ? u[R - 1] : first[b][0][w + 1][lane];
        float2 below2 = lowest ? u[R - 1] : first[b][1][w + 1][lane];
        const float2 above = top ? u[1] : (w > 0 ? last[b][0][w - 1][lane] : u[0]);
        const float2 above_l = top ? u[0] : (w > 0 ? last[b][1][w - 1][lane] : u[0]);
        const float2 above_h = top ? (q.ny == 2 ? u[0] : (R > 2 ? u[R > 2 ? 2 : 0] : below)) : u[0];
        if (q.edge)
            iterate(std::true_type{}, above_l, above, above_h, below, below2, sum);
        else
            iterate(std::false_type{}, above_l, above, above_h, below, below2, sum);
    });
#pragma unroll
    for (int r = 0; r < R; r++) q.store(Un, r, u[r]);
    if (CHECK) store_partial(norms, fr.partials + tile_index<CHECK>(fr));
}

using Kernel = decltype(&k_llt_strip2d<2, false>);
Kernel pick(const Plan& P, bool check) {
    if (P.R == 2) return check ? k_llt_strip2d<2, true> : k_llt_strip2d<2, false>;
    if (P.R == 3) return check ? k_llt_strip2d<3, true> : k_llt_strip2d<3, false>;
    return check ? k_llt_strip2d<4, true> : k_llt_strip2d<4, false>;
}

}  // namespace

bool llt_strip_applies(const Dims& d, bool checking) {
    const char* ek = getenv("CILREG_LLT_KERNEL");
    if (!strip::applies(d) || (ek && ek[0] != '\0')) return false;
    int R, T;
    // k_llt_pair2d, one iteration per graph node, is 1-5% faster for even rows
    // without a stopping rule from 720,000 to 2.1 M pixels (1084x1600 10.7
    // against 11.0 us per iteration; 512^2 3.5 against 2.4, 1500^2 13.5 against
    // 12.2)
    const bool one = d.nx % 2 == 0 && !checking && d.n >= 720000 && d.n < (1LL << 21);
    return !one || strip::forced(&R, &T);
}

int llt_strip_run(const float* f, float* u_out, float lam_rof, float lam_llt, int iters, float tau, float epsil,
                  const Dims& d, cudaStream_t s, float* info) {
    static const Choices choices = {2, 3, {2, 3, 4}, {2, 1, 1}, 1600.0, 850.0};
    return run_flow(choices, f, f, u_out, iters, epsil, d, s, info, true,
                    [&](const Plan& P, bool rule, const Frame& fr, const float* src, float* dst) {
                        return launch_strip(pick(P, rule), P, fr, rule, s, src, dst, f, lam_rof, lam_llt, tau);
                    });
}

}  // namespace cilreg
