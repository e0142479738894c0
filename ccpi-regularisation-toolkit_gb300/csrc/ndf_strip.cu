// Linear / non-linear diffusion on 2D images, several iterations per launch
// (strip2d.cuh), with the arithmetic of k_ndf_pair2d (Diffusion_core.c:
// 140-239).  Every flux is odd in its difference, so the mirrored neighbour at
// an edge of the image is the flux across the opposite face with its sign
// turned: no case of its own beyond the row above row 0, which is row 1.
#include "ndf_tiled.cuh"
#include "strip2d.cuh"

namespace cilreg {

namespace {

using namespace strip;

template <int PEN, int R, bool CHECK>
__global__ void __launch_bounds__(NT, R <= 4 ? 2 : 1)
    k_ndf_strip2d(const float* __restrict__ U, float* __restrict__ Un, const float* __restrict__ F, float lam, float sg,
                  float isg, float tau, Frame fr) {
    __shared__ float2 first[2][NW][32], last[2][NW][32];
    const Place<R> q(fr, CHECK, max(tile_index<CHECK>(fr), 0));
    const int lane = q.lane, w = q.w;
    float2 f[R], u[R];
#pragma unroll
    for (int r = 0; r < R; r++) f[r] = q.load_const(F, r);  // never changes: loaded before the wait
    if (!begin<CHECK>(fr)) return;
#pragma unroll
    for (int r = 0; r < R; r++) u[r] = q.load(U, r);
    const float2 isg2 = splat(isg), lam2 = splat(lam), tau2 = splat(tau);
    Norms norms;

    auto iterate = [&](auto edge_, float2 above, float2 below, auto sum) {
        constexpr bool EDGE = decltype(edge_)::value;
        float2 south = flux2<PEN>(sub2(u[0], above), sg, isg2);
#pragma unroll
        for (int r = 0; r < R; r++) {
            float2 c = u[r];
            float lo, hi;
            x_neighbours<EDGE>(q, c, lo, hi);
            const float2 fx = flux2<PEN>(make_float2(c.y - c.x, hi - c.y), sg, isg2);
            float2 fy = flux2<PEN>(sub2((r < R - 1) ? u[r + 1 < R ? r + 1 : r] : below, c), sg, isg2);
            if (EDGE && r == q.bottom) fy = neg2(south);
            float west = left_of(fx);
            if (EDGE && q.at_left) west = -fx.x;
            // e + w + n + s (Diffusion_core.c:160-164)
            const float2 s = sub2(add2(sub2(fx, make_float2(west, fx.x)), fy), south);
            const float2 t = sub2(c, f[r]);
            const float2 un = fma2(tau2, fma2(lam2, s, neg2(t)), c);
            if (CHECK && sum) add_norms(q, r, un, c, norms);
            u[r] = un;
            south = fy;
        }
    };
    iterations<CHECK>(fr.count, [&](int t, auto sum) {
        const int b = t & 1;
        first[b][w][lane] = u[0];
        last[b][w][lane] = u[R - 1];
        __syncthreads();
        const float2 below = w < NW - 1 ? first[b][w + 1][lane] : u[R - 1];
        const float2 above = q.Y == 0 ? u[1] : (w > 0 ? last[b][w - 1][lane] : u[0]);
        if (q.edge)
            iterate(std::true_type{}, above, below, sum);
        else
            iterate(std::false_type{}, above, below, sum);
    });
#pragma unroll
    for (int r = 0; r < R; r++) q.store(Un, r, u[r]);
    if (CHECK) store_partial(norms, fr.partials + tile_index<CHECK>(fr));
}

using Kernel = decltype(&k_ndf_strip2d<0, 2, false>);
template <int PEN>
Kernel pick_pen(const Plan& P, bool check) {
    if (P.R == 2) return check ? k_ndf_strip2d<PEN, 2, true> : k_ndf_strip2d<PEN, 2, false>;
    if (P.R == 4) return check ? k_ndf_strip2d<PEN, 4, true> : k_ndf_strip2d<PEN, 4, false>;
    return check ? k_ndf_strip2d<PEN, 6, true> : k_ndf_strip2d<PEN, 6, false>;
}
Kernel pick(int pen, const Plan& P, bool check) {
    switch (pen) {
        case 0: return pick_pen<0>(P, check);
        case 1: return pick_pen<1>(P, check);
        case 2: return pick_pen<2>(P, check);
        case 3: return pick_pen<3>(P, check);
        case 4: return pick_pen<4>(P, check);
        default: return pick_pen<5>(P, check);
    }
}

}  // namespace

bool ndf_strip_applies(const Dims& d) {
    const char* ek = getenv("CILREG_NDF_KERNEL");
    return strip::applies(d) && !(ek && ek[0] != '\0');
}

int ndf_strip_run(int pen, const float* f, float* u_out, float lam, float sg, float isg, int iters, float tau,
                  float epsil, const Dims& d, cudaStream_t s, float* info, const float* u_init) {
    static const Choices choices = {1, 3, {2, 4, 6}, {2, 2, 1}, 500.0, 250.0};
    return run_flow(choices, f, u_init ? u_init : f, u_out, iters, epsil, d, s, info, true,
                    [&](const Plan& P, bool rule, const Frame& fr, const float* src, float* dst) {
                        return launch_strip(pick(pen, P, rule), P, fr, rule, s, src, dst, f, lam, sg, isg, tau);
                    });
}

}  // namespace cilreg
