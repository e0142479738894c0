// Fourth-order diffusion on 2D images, several iterations per launch
// (strip2d.cuh), with the arithmetic of k_d4_pair2d
// (Diffus4th_order_core.c:136-265).  The weighted Laplacian W costs three
// quarters of an iteration, so the rows of W above and below a strip are
// exchanged after a second barrier instead of being recomputed.
#include "diff4th_tiled.cuh"
#include "strip2d.cuh"

namespace cilreg {

namespace {

using namespace strip;

template <int R, bool CHECK>
__global__ void __launch_bounds__(NT, R <= 2 ? 2 : 1)
    k_d4_strip2d(const float* __restrict__ U, float* __restrict__ Un, const float* __restrict__ F, float lam, float tau,
                 float isg2, Frame fr) {
    __shared__ float2 firstU[NW][32], lastU[NW][32], firstW[NW][32], lastW[NW][32];
    const Place<R> q(fr, CHECK, max(tile_index<CHECK>(fr), 0));
    const int lane = q.lane, w = q.w;
    const float EPS = 1.0e-7f;
    const float2 HALF2 = splat(0.5f), QUART2 = splat(0.25f), TWO2 = splat(2.0f), MTWO2 = splat(-2.0f);
    const float2 ONE2 = splat(1.0f), isg22 = splat(isg2), tau2 = splat(tau), mlam2 = splat(-lam);
    float2 f[R], u[R];
#pragma unroll
    for (int r = 0; r < R; r++) f[r] = q.load_const(F, r);  // never changes: loaded before the wait
    if (!begin<CHECK>(fr)) return;
#pragma unroll
    for (int r = 0; r < R; r++) u[r] = q.load(U, r);
    Norms norms;

    struct Row {
        float2 c, lo, hi;  // the pair, (x-1, x) and (x+1, x+2)
    };
    float2 W[R];
    auto laplacian = [&](auto edge_, float2 above, float2 below) {
        constexpr bool EDGE = decltype(edge_)::value;
        auto row_of = [&](float2 c) -> Row {
            float lo, hi;
            x_neighbours<EDGE>(q, c, lo, hi);
            return Row{c, make_float2(lo, c.x), make_float2(c.y, hi)};
        };
        Row m = row_of(above), c = row_of(u[0]);
#pragma unroll
        for (int r = 0; r < R; r++) {
            const Row next = row_of((r < R - 1) ? u[r + 1 < R ? r + 1 : r] : below);
            const Row h = (EDGE && r == q.bottom) ? m : next;
            const float2 gx = mul2(HALF2, sub2(c.lo, c.hi));
            const float2 gy = mul2(HALF2, sub2(m.c, h.c));
            const float2 gx2 = mul2(gx, gx), gy2 = mul2(gy, gy);
            const float2 gxx = fma2(MTWO2, c.c, add2(c.lo, c.hi));
            const float2 gyy = fma2(MTWO2, c.c, add2(m.c, h.c));
            const float2 gxy = mul2(QUART2, sub2(sub2(add2(m.lo, h.hi), h.lo), m.hi));
            const float2 xy2 = mul2(mul2(mul2(TWO2, gx), gy), gxy);
            const float2 den = add2(gx2, gy2);
            const float2 nn = fma2(gyy, gy2, fma2(gxx, gx2, xy2));
            const float2 oo = fma2(gyy, gx2, fma2(gxx, gy2, neg2(xy2)));
            const float2 iq = rcp2(make_float2((den.x <= EPS) ? EPS : den.x, (den.y <= EPS) ? EPS : den.y));
            const float2 vn = mul2(nn, iq), vo = mul2(oo, iq);
            const float2 cc = rcp2(fma2(den, isg22, ONE2));
            W[r] = fma2(mul2(cc, cc), vn, mul2(cc, vo));
            m = c;
            c = next;
        }
    };
    auto update = [&](auto edge_, float2 wm, float2 wbelow, auto sum) {
        constexpr bool EDGE = decltype(edge_)::value;
#pragma unroll
        for (int r = 0; r < R; r++) {
            float2 wc = W[r];
            float lo, hi;
            x_neighbours<EDGE>(q, wc, lo, hi);
            float2 wh = (r < R - 1) ? W[r + 1 < R ? r + 1 : r] : wbelow;
            if (EDGE && r == q.bottom) wh = wm;
            const float2 lx = fma2(MTWO2, wc, add2(make_float2(lo, wc.x), make_float2(wc.y, hi)));
            const float2 ly = fma2(MTWO2, wc, add2(wm, wh));
            const float2 lap = add2(lx, ly);
            const float2 un = fma2(tau2, fma2(mlam2, lap, neg2(sub2(u[r], f[r]))), u[r]);
            if (CHECK && sum) add_norms(q, r, un, u[r], norms);
            u[r] = un;
            wm = W[r];
        }
    };
    iterations<CHECK>(fr.count, [&](int t, auto sum) {
        firstU[w][lane] = u[0];
        lastU[w][lane] = u[R - 1];
        __syncthreads();
        const float2 below = w < NW - 1 ? firstU[w + 1][lane] : u[R - 1];
        const float2 above = q.Y == 0 ? u[1] : (w > 0 ? lastU[w - 1][lane] : u[0]);
        if (q.edge)
            laplacian(std::true_type{}, above, below);
        else
            laplacian(std::false_type{}, above, below);
        firstW[w][lane] = W[0];
        lastW[w][lane] = W[R - 1];
        __syncthreads();
        const float2 wbelow = w < NW - 1 ? firstW[w + 1][lane] : W[R - 1];
        const float2 wabove = q.Y == 0 ? W[1] : (w > 0 ? lastW[w - 1][lane] : W[0]);
        if (q.edge)
            update(std::true_type{}, wabove, wbelow, sum);
        else
            update(std::false_type{}, wabove, wbelow, sum);
    });
#pragma unroll
    for (int r = 0; r < R; r++) q.store(Un, r, u[r]);
    if (CHECK) store_partial(norms, fr.partials + tile_index<CHECK>(fr));
}

using Kernel = decltype(&k_d4_strip2d<2, false>);
Kernel pick(const Plan& P, bool check) {
    if (P.R == 2) return check ? k_d4_strip2d<2, true> : k_d4_strip2d<2, false>;
    if (P.R == 3) return check ? k_d4_strip2d<3, true> : k_d4_strip2d<3, false>;
    return check ? k_d4_strip2d<4, true> : k_d4_strip2d<4, false>;
}

}  // namespace

bool d4_strip_applies(const Dims& d) {
    const char* ek = getenv("CILREG_D4_KERNEL");
    return strip::applies(d) && !(ek && ek[0] != '\0');
}

int d4_strip_run(const float* f, float* u_out, float lam, int iters, float tau, float isg2, float epsil, const Dims& d,
                 cudaStream_t s, float* info) {
    static const Choices choices = {2, 3, {2, 3, 4}, {2, 1, 1}, 870.0, 420.0};
    return run_flow(choices, f, f, u_out, iters, epsil, d, s, info, true,
                    [&](const Plan& P, bool rule, const Frame& fr, const float* src, float* dst) {
                        return launch_strip(pick(P, rule), P, fr, rule, s, src, dst, f, lam, tau, isg2);
                    });
}

}  // namespace cilreg
