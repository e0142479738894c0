// ROF-TV on 2D images, several iterations per launch (strip2d.cuh).
//
// The arithmetic is k_rof_pair2d's, operation by operation (ROF_TV_core.c:
// 102-160).  An iteration of a strip needs one row of U above and below it;
// the y flux D1 of the row above is recomputed from that row.
#include "drivers.cuh"
#include "nvtx.cuh"
#include "rof_tiled.cuh"
#include "strip2d.cuh"

namespace cilreg {

namespace {

using namespace strip;

// ONCE: the result is only used by one subtraction
template <bool ONCE = false>
__device__ __forceinline__ float2 normalise2(float2 dp, float2 s) {
    const float2 r = make_float2(rsqrt_normal(s.x), rsqrt_normal(s.y));
    return ONCE ? mul2_rn(dp, r) : mul2(dp, r);
}

template <int R, bool CHECK, bool LARR>
__global__ void __launch_bounds__(NT, R <= 4 ? 2 : 1)
    k_rof_strip2d(const float* __restrict__ U, float* __restrict__ Un, const float* __restrict__ F,
                  const float* __restrict__ lam_arr, float lam, float tau, Frame fr) {
    __shared__ float2 first[2][NW][32], last[2][NW][32];
    const Place<R> q(fr, CHECK, max(tile_index<CHECK>(fr), 0));
    const int lane = q.lane, w = q.w, Y = q.Y;
    // f and the lambda map never change during a run: loaded before waiting
    // for the previous launch (launch_pdl)
    float2 f[R], l[LARR ? R : 1], u[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
        f[r] = q.load_const(F, r);
        if (LARR) l[r] = q.load_const(lam_arr, r);
    }
    if (!LARR) l[0] = splat(lam);
    if (!begin<CHECK>(fr)) return;
#pragma unroll
    for (int r = 0; r < R; r++) u[r] = q.load(U, r);
    const float2 EPS2 = splat(1.0e-8f), tau2 = splat(tau);
    Norms norms;

    // above: the row over the strip (the mirrored row 1 over row 0), next: the
    // row under that one
    auto iterate = [&](auto edge_, float2 above, float2 next, float2 below, auto sum) {
        constexpr bool EDGE = decltype(edge_)::value;
        // squared minmod of the x differences of a row, and its forward difference
        auto along_x = [&](float2& c, float2& xp, float2& mx2) {
            float lo, hi;
            x_neighbours<EDGE>(q, c, lo, hi);
            const float dxc = c.y - c.x;
            xp = make_float2(dxc, hi - c.y);
            mx2 = minmod_sq2(xp, make_float2(c.x - lo, dxc));
        };
        float2 d1l;  // D1 of the row above
        {
            float2 c = above, xp, mx2;
            along_x(c, xp, mx2);
            const float2 yp = sub2(next, c);
            d1l = normalise2(yp, add2(fma2(yp, yp, mx2), EPS2));
        }
        float2 ym = sub2(u[0], above);
#pragma unroll
        for (int r = 0; r < R; r++) {
            float2 c = u[r], xp, mx2;
            const float2 dn = (r < R - 1) ? u[r + 1 < R ? r + 1 : r] : below;
            float2 yp = sub2(dn, c);
            if (EDGE && r == q.bottom) yp = neg2(ym);  // mirrored: the row above is also the row below
            along_x(c, xp, mx2);
            const float2 my2 = minmod_sq2(yp, ym);
            const float2 s1 = add2(fma2(yp, yp, mx2), EPS2);
            const float2 d1 = (r == R - 1) ? normalise2<true>(yp, s1) : normalise2(yp, s1);
            const float2 d2 = normalise2(xp, add2(fma2(xp, xp, my2), EPS2));
            float d2l = left_of(d2);
            if (EDGE && q.at_left) d2l = d2.y;
            const float2 div = add2(sub2(d1, d1l), sub2(d2, make_float2(d2l, d2.x)));
            const float2 t = sub2(c, f[r]);
            const float2 un = fma2(tau2, fma2(l[LARR ? r : 0], div, neg2(t)), c);
            if (CHECK && sum) add_norms(q, r, un, c, norms);
            u[r] = un;
            ym = yp;
            d1l = d1;
        }
    };
    iterations<CHECK>(fr.count, [&](int t, auto sum) {
        const int b = t & 1;
        first[b][w][lane] = u[0];
        last[b][w][lane] = u[R - 1];
        __syncthreads();
        const float2 below = w < NW - 1 ? first[b][w + 1][lane] : u[R - 1];
        const float2 above = Y == 0 ? u[1] : (w > 0 ? last[b][w - 1][lane] : u[0]);
        const float2 next = Y == 0 ? (R > 2 ? u[R > 2 ? 2 : 0] : below) : u[0];
        if (q.edge)
            iterate(std::true_type{}, above, q.ny == 2 && Y == 0 ? u[0] : next, below, sum);
        else
            iterate(std::false_type{}, above, next, below, sum);
    });
#pragma unroll
    for (int r = 0; r < R; r++) q.store(Un, r, u[r]);
    if (CHECK) store_partial(norms, fr.partials + tile_index<CHECK>(fr));
}

using Kernel = decltype(&k_rof_strip2d<2, false, false>);
template <int R>
Kernel pick_r(bool check, bool larr) {
    return check ? (larr ? k_rof_strip2d<R, true, true> : k_rof_strip2d<R, true, false>)
                 : (larr ? k_rof_strip2d<R, false, true> : k_rof_strip2d<R, false, false>);
}
Kernel pick(const Plan& P, bool check, bool larr) {
    return P.R == 2 ? pick_r<2>(check, larr) : P.R == 3 ? pick_r<3>(check, larr)
         : P.R == 4 ? pick_r<4>(check, larr) : pick_r<6>(check, larr);
}

}  // namespace

bool rof_strip_applies(const Dims& d) {
    const char* ek = getenv("CILREG_ROF_KERNEL");
    return strip::applies(d) && !(ek && ek[0] != '\0');
}

int rof_strip_run(const float* f, float* u_out, const float* lam_arr, float lam, int iters, float tau, float epsil,
                  const Dims& d, cudaStream_t s, float* info, const float* u_init) {
    static const Choices choices = {1, 4, {2, 3, 4, 6}, {2, 2, 2, 1}, 660.0, 300.0};
    const bool larr = lam_arr != nullptr;
    return run_flow(choices, f, u_init ? u_init : f, u_out, iters, epsil, d, s, info, !larr || host_aligned8(lam_arr),
                    [&](const Plan& P, bool rule, const Frame& fr, const float* src, float* dst) {
                        return launch_strip(pick(P, rule, larr), P, fr, rule, s, src, dst, f, lam_arr, lam, tau);
                    });
}

}  // namespace cilreg
