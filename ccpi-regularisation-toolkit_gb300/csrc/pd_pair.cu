// PD-TV iteration of a 3D volume with two voxels per thread along x (reference
// arithmetic PD_TV_core.c:212-252, with k_pd_stream's roundings).
//
// k_pd_stream is bound by instruction issue (133 us per 256^3 iteration, whose
// 36 B per voxel take 89): the exact projection and division, the shared-memory
// exchange and the addresses of every voxel.  Here, as in k_rof_pair, the
// differences and sums of two voxels issue paired, one address and one loop
// serve both, and the x neighbours (Ue(x+2), P1(x-1)) come by shuffles from the
// neighbouring thread, so that shared memory serves the y neighbours alone.
// Products that feed one addition stay scalar (mul2_rn): the iterates are
// k_pd_stream's bit for bit.
//
// Time per iteration, k_pd_stream -> this: 96^3 11.6 -> 8.7 us, 192^3 63 -> 54,
// 256^3 134 -> 115, 512^3 993 -> 887 (711 at the copy rate), 143x201x255 61 ->
// 58.  Tried and slower: 24 rows (512^3 893, 256^3 121, 96^3 10.8), 32 rows
// (1023), three CTAs per SM at 80 registers (1041), five at 48 (919).
//
// Thread tx of a row holds the pair (X, X+1), X even; a CTA of 16 x 16 threads
// updates the pairs of threads 1..15 and rows 1..14 (the last thread loads its
// upper x neighbour itself, so that only one pair per row is halo).  Step j:
//   A. forms and projects P'(j-1) and publishes its y component;
//   B. publishes Ue(j) (loaded one step earlier);
//   C. after one barrier, updates plane j-1 and writes Ue', P'.
// Odd rows (a last pair whose second voxel is the mirrored one) and arrays off
// 8-byte alignment run the 4-byte instantiation.
#include <stdlib.h>

#include "pair.cuh"
#include "pd_tiled.cuh"

namespace cilreg {

namespace {

using namespace pair;

constexpr int LX = 16, ROWS = 16;
constexpr int OXD = 2 * (LX - 1);           // updated voxels along x
constexpr int OYD = ROWS - 2;
constexpr int NTD = LX * ROWS, TPD = 2 * NTD;
constexpr int ZCHUNK = 64;

template <bool CHECK, bool ALIGNED>
__global__ void __launch_bounds__(NTD, 4) k_pd_pair(PdStreamArgs a, Dims d, int zc, const StopCtl* ctl,
                                                    double2* partials) {
    __shared__ __align__(16) float sU[2][TPD];
    __shared__ __align__(16) float sP[2][TPD];
    pdl_wait();  // the previous iteration has completed (launch_pdl)
    if (pdl_many_waves()) pdl_trigger();
    if (ctl->stop) return;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int nx = d.nx, ny = d.ny, nz = d.nz;
    const int X = blockIdx.x * OXD - 2 + 2 * tx;  // x of the pair's first voxel
    const int y = blockIdx.y * OYD - 1 + ty;
    const bool upd = tx >= 1 && ty >= 1 && ty <= ROWS - 2 && X < nx && y < ny;
    const bool x_last = X + 2 == nx;
    const bool oend = !ALIGNED && X + 1 == nx;  // the pair's first voxel ends an odd row
    // upper y neighbour in the tile (mirrored at the volume's edge, clamped
    // where only unused halo values depend on it)
    int yh = (ny == 1) ? ty : ((y + 1 >= ny) ? ty - 1 : ty + 1);
    yh = min(max(yh, 0), ROWS - 1);
    const int o = (ty * LX + tx) * 2, oyh = (yh * LX + tx) * 2, oyl = (max(ty - 1, 0) * LX + tx) * 2;
    const int row = min(max(y, 0), ny - 1) * nx;
    const int col = row + (ALIGNED ? min(max(X, 0), nx - 2) : pair_col(X, nx));
    const int dc = ALIGNED ? 1 : pair_step(X, nx);
    const int colr = row + min(X + 2, nx - 1);  // of the last thread's upper x neighbour
    const bool last = tx == LX - 1;
    const float2 sigma2 = splat(a.sigma), tau2 = splat(a.tau), lt2 = splat(a.lt);
    float2 pa = splat(0.f), pb = splat(0.f);
    const int z0 = blockIdx.z * zc;
    const int z1 = min(z0 + zc, nz);
    const int sxy = (int)d.sxy;
    auto plane = [&](int k) -> int { return min(max(k, 0), nz - 1) * sxy; };
    auto ldg2 = [&](const float* p) -> float2 {
        if (ALIGNED) return __ldg(reinterpret_cast<const float2*>(p));
        return make_float2(__ldg(p), __ldg(p + dc));
    };
    auto put = [&](float* p, float2 v) {
        if (ALIGNED) {
            st2(p, v);
        } else {
            p[0] = v.x;
            if (!oend) p[1] = v.y;
        }
    };
    // registers entering step j: Ue of planes j-2, j-1, j (and the last
    // thread's upper neighbour), the old dual and f of plane j-1
    float2 um2 = ldg2(a.u + plane(z0 - 2) + col), um1 = ldg2(a.u + plane(z0 - 1) + col),
           uj = ldg2(a.u + plane(z0) + col);
    float rm1 = last ? __ldg(a.u + plane(z0 - 1) + colr) : 0.f, rj = last ? __ldg(a.u + plane(z0) + colr) : 0.f;
    float2 q[3], fq = ldg2(a.f + plane(z0 - 1) + col);
#pragma unroll
    for (int c = 0; c < 3; c++) q[c] = ldg2(a.p[c] + plane(z0 - 1) + col);
    float2 p3m = splat(0.f);  // projected z component of the previous plane
    st2(sU[1] + o, um1);      // slot of plane p: (p - z0) & 1
    __syncthreads();

    auto step = [&](auto par, int j) {
        constexpr int P = decltype(par)::value;  // (j - z0) & 1
        const int k = j - 1;                     // plane of this step's dual and update
        // prefetch for the next step: Ue(j+1), old dual and f of plane j
        const int ou = plane(min(j + 1, z1)), oj = plane(j);
        const float2 un1 = ldg2(a.u + ou + col);
        const float rn = last ? __ldg(a.u + ou + colr) : 0.f;
        float2 nq[3];
#pragma unroll
        for (int c = 0; c < 3; c++) nq[c] = ldg2(a.p[c] + oj + col);
        const float2 nf = ldg2(a.f + oj + col);
        // A. projected dual of plane k
        float2 p[3];
        {
            const float2 c = um1;
            float hi = __shfl_down_sync(0xffffffffu, c.x, 1, LX);
            hi = x_last ? c.x : last ? rm1 : hi;
            const float2 zhi = (k + 1 >= nz) ? um2 : uj;  // mirrored (PD_TV_core.c:225)
            p[0] = add2(q[0], mul2_rn(sigma2, sub2(make_float2(c.y, hi), c)));
            p[1] = add2(q[1], mul2_rn(sigma2, sub2(ld2(sU[1 - P] + oyh), c)));
            p[2] = add2(q[2], mul2_rn(sigma2, sub2(zhi, c)));
            if (!a.aniso) {
                const float2 den = add2(add2(mul2_rn(p[0], p[0]), mul2_rn(p[1], p[1])), mul2_rn(p[2], p[2]));
                if (den.x > 1.0f) {
                    const float s = __fdiv_rn(1.0f, __fsqrt_rn(den.x));
#pragma unroll
                    for (int i = 0; i < 3; i++) p[i].x = __fmul_rn(p[i].x, s);
                }
                if (den.y > 1.0f) {
                    const float s = __fdiv_rn(1.0f, __fsqrt_rn(den.y));
#pragma unroll
                    for (int i = 0; i < 3; i++) p[i].y = __fmul_rn(p[i].y, s);
                }
            } else {
#pragma unroll
                for (int i = 0; i < 3; i++) p[i] = make_float2(unit_clip(p[i].x), unit_clip(p[i].y));
            }
            st2(sP[1 - P] + o, p[1]);
        }
        float lo = __shfl_up_sync(0xffffffffu, p[0].y, 1, LX);
        // B. publish Ue(j)
        st2(sU[P] + o, uj);
        __syncthreads();
        // C. primal update of plane k
        if (upd && k >= z0) {
            if (X == 0) lo = 0.f;
            const float2 yl = (y == 0) ? splat(0.f) : ld2(sP[1 - P] + oyl);
            const float2 zl = (k == 0) ? splat(0.f) : p3m;
            // div = -(P1 - P1[-1]) - (P2 - P2[-1]) - (P3 - P3[-1]), P[-1] = 0
            float2 dv = add2(sub2(make_float2(lo, p[0].x), p[0]), sub2(yl, p[1]));
            dv = add2(dv, sub2(zl, p[2]));
            float2 uc = um1;
            if (a.nonneg) uc = make_float2(uc.x < 0.f ? 0.f : uc.x, uc.y < 0.f ? 0.f : uc.y);
            const float2 num = add2(sub2(uc, mul2_rn(tau2, dv)), mul2_rn(lt2, fq));
            const float2 un = div_by_double2(num, a.onelt);
            const int v = k * sxy + col;
            if (CHECK) {
                const float2 df = sub2(un, uc);
                const float2 dm = make_float2(df.x, oend ? 0.f : df.y), um = make_float2(un.x, oend ? 0.f : un.y);
                pa = fma2(dm, dm, pa);
                pb = fma2(um, um, pb);
                put(a.ubrk + v, un);
            }
            put(a.un + v, add2(un, mul2_rn(splat(a.theta), sub2(un, uc))));
#pragma unroll
            for (int c = 0; c < 3; c++) put(a.pn[c] + v, p[c]);
        }
        p3m = p[2];
        um2 = um1;
        um1 = uj;
        uj = un1;
        rm1 = rj;
        rj = rn;
#pragma unroll
        for (int c = 0; c < 3; c++) q[c] = nq[c];
        fq = nf;
    };
    int j = z0;
    for (; j + 1 <= z1; j += 2) {
        step(Ic<0>{}, j);
        step(Ic<1>{}, j + 1);
    }
    if (j <= z1) step(Ic<0>{}, j);
    if (!pdl_many_waves()) pdl_trigger();
    if (CHECK) block_pair_partial<NTD>(pa.x + pa.y, pb.x + pb.y, partials, block_slot());
}

using Kernel = decltype(&k_pd_pair<false, true>);
Kernel pick(bool check, bool aligned) {
    if (aligned) return check ? k_pd_pair<true, true> : k_pd_pair<false, true>;
    return check ? k_pd_pair<true, false> : k_pd_pair<false, false>;
}

}  // namespace

PdPlan pd_pair_plan(const Dims& d, bool aligned) {
    PdPlan T;
    const char* e = getenv("CILREG_PD_KERNEL");
    // "stream" (or "simple") keeps a one-voxel kernel
    T.pair = d.nz > 1 && pair_rows(d) && !(e && e[0] != '\0');
    if (!T.pair) return T;
    T.aligned = aligned && d.nx % 2 == 0;
    T.block = dim3(LX, ROWS, 1);
    static const int resident = resident_ctas(k_pd_pair<false, true>, NTD);
    const int gx = (d.nx + OXD - 1) / OXD, gy = (d.ny + OYD - 1) / OYD;
    T.zchunk = wave_zchunk((long long)gx * gy, d.nz, resident, 1, ZCHUNK, 2.5);
    T.grid = dim3(gx, gy, (d.nz + T.zchunk - 1) / T.zchunk);
    T.nblocks = (long long)T.grid.x * T.grid.y * T.grid.z;
    return T;
}

int pd_pair_step(const PdPlan& T, const PdStreamArgs& a, const Dims& d, const StopCtl* ctl, double2* partials,
                 cudaStream_t s) {
    CILREG_CUDA(launch_pdl(pick(a.check != 0, T.aligned), T.grid, T.block, 0, s, a, d, T.zchunk, ctl, partials));
    return OK;
}
}  // namespace cilreg
