// Split-Bregman outer iteration k >= 1 with two voxels per thread along x
// (reference arithmetic SB_TV_core.c:254-371): 3D volumes.
//
// The pass of k_sb_fused (state U^k and B^{k-1}; D^k, B^k formed on the fly,
// both Jacobi sweeps, 36 B per voxel) is bound by the issue of its
// instructions: 36 B take 89 us at 256^3, it took 201.  Here a thread's work is
// doubled along x, as in k_rof_pair: FP32 arithmetic issues paired, one address
// and one loop serve two voxels.  D and B enter a sweep only by D - B, which
// takes their place in the exchange; its x neighbours, U's and U1's come by
// shuffles from the neighbouring thread's registers, and shared memory serves
// the y neighbours alone (6 8-byte loads and 3 stores per pair and plane,
// against 18 and 6 4-byte ones per voxel).  |v| and 1/|v| share one approximate
// reciprocal square root, refined paired, in place of an IEEE square root and
// an IEEE reciprocal per voxel.
//
// Time per iteration, k_sb_fused -> this: 64^3 9.1 -> 7.2 us, 96^3 15.6 ->
// 10.6, 192^3 86 -> 64, 256^3 201 -> 147, 512^3 1427 -> 1091 (711 at the copy
// rate), 143x201x255 97 -> 83, 511^3 1436 -> 1302.  Tried and slower: copies to shared memory two planes ahead by cp.async
// (256^3 190), loads issued after the shrinkage (170 to 195), one CTA of 32 rows
// per SM (180), three of 16 (154), 16 rows at 128 registers (181).
//
// Thread tx of a row holds the pair (X, X+1), X even; a CTA of LX x ROWS
// threads updates whole pairs, threads 1..LX-2 of rows 2..ROWS-3.  Step j:
//   A0. forms D^k, B^k of plane j-1 (y successors of U^k from shared memory, k
//       successor from registers); publishes Dy - By; writes B^k;
//   A.  forms G and U1 of plane j-2 and publishes U1;
//   B.  forms U2 of plane j-3 and writes it;
//   C.  publishes U^k of plane j (loaded one step earlier).
// One barrier per plane.  Odd rows (a last pair whose second voxel is the
// mirrored one) and arrays off 8-byte alignment run the 4-byte instantiation.
#include <stdlib.h>

#include "pair.cuh"
#include "sb_tiled.cuh"

namespace cilreg {

namespace {

using namespace pair;

constexpr int LX = 16;
constexpr int OXS = 2 * LX - 4;
constexpr int ZCHUNK = 64;

template <bool CHECK, bool ANISO, bool ALIGNED, int ROWS>
__global__ void __launch_bounds__(LX * ROWS, 2) k_sb_pair(SbFusedArgs a, Dims d, int zc, const StopCtl* ctl,
                                                          double2* partials) {
    constexpr int OYS = ROWS - 4, NTS = LX * ROWS, TPS = 2 * NTS;
    __shared__ __align__(16) float sU[4][TPS];
    __shared__ __align__(16) float sU1[2][TPS];
    __shared__ __align__(16) float sQ[2][TPS];
    pdl_wait();  // the previous iteration has completed (launch_pdl)
    if (pdl_many_waves()) pdl_trigger();
    if (ctl->stop) return;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int nx = d.nx, ny = d.ny, nz = d.nz;
    const int X = blockIdx.x * OXS - 2 + 2 * tx;  // x of the pair's first voxel
    const int y = blockIdx.y * OYS - 2 + ty;
    const bool upd = tx >= 1 && tx <= LX - 2 && ty >= 2 && ty <= ROWS - 3 && X >= 0 && X < nx && y >= 0 && y < ny;
    const bool x_first = X == 0, x_last = X + 2 == nx;
    const bool oend = !ALIGNED && X + 1 == nx;  // the pair's first voxel ends an odd row
    // y neighbours in the tile (mirrored at the volume's edges, clamped where
    // only unused halo values depend on them; a row of length 1 maps to itself)
    int yl = (ny == 1) ? ty : ((y - 1 < 0) ? ty + 1 : ty - 1);
    int yh = (ny == 1) ? ty : ((y + 1 >= ny) ? ty - 1 : ty + 1);
    yl = min(max(yl, 0), ROWS - 1);
    yh = min(max(yh, 0), ROWS - 1);
    const int o = (ty * LX + tx) * 2, oyl = (yl * LX + tx) * 2, oyh = (yh * LX + tx) * 2;
    const int col = min(max(y, 0), ny - 1) * nx + (ALIGNED ? min(max(X, 0), nx - 2) : pair_col(X, nx));
    const int dc = ALIGNED ? 1 : pair_step(X, nx);
    const float2 lam2 = splat(a.lambda), mu2 = splat(a.mu), nrm2 = splat(a.norm);
    const float dlam = a.dlam;
    float2 pa = splat(0.f), pb = splat(0.f);
    const int z0 = blockIdx.z * zc;
    const int z1 = min(z0 + zc, nz);
    const int sxy = (int)d.sxy;
    auto at = [&](int k) -> int { return min(max(k, 0), nz - 1) * sxy + col; };
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
    // (x-1, x) and (x+1, x+2) of a pair: mirrored at the volume's edges (a
    // tile's outermost threads see their own values: unused halo)
    auto below = [&](float2 c) -> float2 {
        const float v = __shfl_up_sync(0xffffffffu, c.y, 1, LX);
        return make_float2(x_first ? c.y : v, c.x);
    };
    auto above = [&](float2 c) -> float2 {
        const float v = __shfl_down_sync(0xffffffffu, c.x, 1, LX);
        return make_float2(c.y, x_last ? c.x : v);
    };
    // registers entering step j: U^k of planes j, j-1, j-2, j-3; B^{k-1} of
    // plane j-1; D, B (x and z components) of plane j-2, z also of j-3; G of
    // plane j-3; U1 of planes j-3, j-4; mu f of planes j-2, j-3
    float2 cu = ldg2(a.u + at(z0 - 1)), pu = ldg2(a.u + at(z0 - 2)), ppu = ldg2(a.u + at(z0 - 3));
    float2 pppu = splat(0.f);
    float2 cb[3];
#pragma unroll
    for (int c = 0; c < 3; c++) cb[c] = ldg2(a.bp[c] + at(z0 - 2));
    float2 qb[3], qzc = splat(0.f);
#pragma unroll
    for (int c = 0; c < 3; c++) qb[c] = splat(0.f);
    float2 gc = splat(0.f), u1c = splat(0.f), u1d = splat(0.f);
    float2 fb = mul2(mu2, ldg2(a.f + at(z0 - 3))), fc = splat(0.f);
    // U ring slot of plane p: (p - z0 + 4) & 3; D/B and U1 slots: (p - z0 + 4) & 1
    st2(sU[2] + o, pu);  // plane z0-2
    __syncthreads();

    // R = (j - z0 + 1) & 3 for step j (steps start at j = z0 - 1)
    auto step = [&](auto rr, auto full, int j) {
        constexpr int R = decltype(rr)::value;
        constexpr bool FULL = decltype(full)::value;
        constexpr int SJ = (R + 3) & 3, SM1 = (R + 2) & 3, SM2 = (R + 1) & 3;  // U slots of j, j-1, j-2
        constexpr int W1 = (R + 2) & 1, W2 = (R + 1) & 1, W3 = R & 1;         // parity slots of j-1, j-2, j-3
        const float2 nu = ldg2(a.u + at(j + 1));
        const int ob = at(j);
        float2 nb[3];
#pragma unroll
        for (int c = 0; c < 3; c++) nb[c] = ldg2(a.bp[c] + ob);
        const float2 nf = ldg2(a.f + at(j - 1));
        // A0. D^k, B^k of plane m0 = j-1
        float2 qa[3];
        {
            float2 da[3], ba[3];
            const int m0 = j - 1;
            const float2 zhi = (m0 == nz - 1) ? ppu : cu;  // mirrored k+1 (SB_TV_core.c:293)
            const float2 gr[3] = {sub2(above(pu), pu), sub2(ld2(sU[SM1] + oyh), pu), sub2(zhi, pu)};
            sb_shrink2(gr, cb, dlam, ANISO, da, ba);
            if (upd && m0 >= z0 && m0 < z1) {
                const int v = m0 * sxy + col;
#pragma unroll
                for (int c = 0; c < 3; c++) put(a.bn[c] + v, ba[c]);
            }
#pragma unroll
            for (int c = 0; c < 3; c++) qa[c] = sub2(da[c], ba[c]);
            st2(sQ[W1] + o, qa[1]);
        }
        // A. G and U1 of plane m = j-2 (SB_TV_core.c:273-280); its Dy, By were
        // published in the previous step
        const int m = j - 2;
        float2 g = sub2(below(qb[0]), qb[0]);
        g = sub2(add2(g, ld2(sQ[W2] + oyl)), qb[1]);
        g = sub2(add2(g, (m == 0) ? qa[2] : qzc), qb[2]);  // mirrored k-1
        const float2 zh0 = (m == nz - 1) ? pppu : pu, zl0 = (m == 0) ? pu : pppu;
        float2 q = add2(above(ppu), below(ppu));
        q = add2(add2(q, ld2(sU[SM2] + oyh)), ld2(sU[SM2] + oyl));
        q = add2(add2(q, zh0), zl0);
        const float2 u1 = mul2(nrm2, fma2(add2(g, q), lam2, fb));
        st2(sU1[W2] + o, u1);
        // B. U2 of plane kf = j-3
        if (FULL) {
            const int kf = j - 3;
            const float2 zh1 = (kf == nz - 1) ? u1d : u1, zl1 = (kf == 0) ? u1 : u1d;
            const float2 xl = below(u1c);
            float2 xh = above(u1c);
            if (oend) xh.x = xl.x;  // the mirrored voxel's own U1 was not formed
            float2 p = add2(xh, xl);
            p = add2(add2(p, ld2(sU1[W3] + oyh)), ld2(sU1[W3] + oyl));
            p = add2(add2(p, zh1), zl1);
            const float2 u2 = mul2(nrm2, fma2(add2(gc, p), lam2, fc));
            if (upd) {
                put(a.u2 + (kf * sxy + col), u2);
                if (CHECK) {
                    const float2 df = sub2(u2, u1c);
                    const float2 dm = make_float2(df.x, oend ? 0.f : df.y), um = make_float2(u2.x, oend ? 0.f : u2.y);
                    pa = fma2(dm, dm, pa);
                    pb = fma2(um, um, pb);
                }
            }
        }
        // C. publish U^k of plane j
        st2(sU[SJ] + o, cu);
        __syncthreads();
        pppu = ppu;
        ppu = pu;
        pu = cu;
        cu = nu;
        qzc = qb[2];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            cb[c] = nb[c];
            qb[c] = qa[c];
        }
        gc = g;
        u1d = u1c;
        u1c = u1;
        fc = fb;
        fb = mul2(mu2, nf);
    };
    step(Ic<0>{}, std::false_type{}, z0 - 1);
    step(Ic<1>{}, std::false_type{}, z0);
    step(Ic<2>{}, std::false_type{}, z0 + 1);
    step(Ic<3>{}, std::false_type{}, z0 + 2);
    int j = z0 + 3;
    for (; j + 3 <= z1 + 2; j += 4) {
        step(Ic<0>{}, std::true_type{}, j);
        step(Ic<1>{}, std::true_type{}, j + 1);
        step(Ic<2>{}, std::true_type{}, j + 2);
        step(Ic<3>{}, std::true_type{}, j + 3);
    }
    if (j <= z1 + 2) step(Ic<0>{}, std::true_type{}, j);
    if (j + 1 <= z1 + 2) step(Ic<1>{}, std::true_type{}, j + 1);
    if (j + 2 <= z1 + 2) step(Ic<2>{}, std::true_type{}, j + 2);
    if (!pdl_many_waves()) pdl_trigger();
    if (CHECK) block_pair_partial<NTS>(pa.x + pa.y, pb.x + pb.y, partials, block_slot());
}

using Kernel = decltype(&k_sb_pair<false, false, true, 24>);
template <int ROWS, bool ALIGNED>
Kernel pick(bool check, bool aniso) {
    if (check) return aniso ? k_sb_pair<true, true, ALIGNED, ROWS> : k_sb_pair<true, false, ALIGNED, ROWS>;
    return aniso ? k_sb_pair<false, true, ALIGNED, ROWS> : k_sb_pair<false, false, ALIGNED, ROWS>;
}

}  // namespace

SbPlan sb_pair_plan(const Dims& d, bool aligned) {
    SbPlan T;
    const char* e = getenv("CILREG_SB_KERNEL");
    // "tiled" keeps the one-voxel kernel
    T.use = d.nz > 1 && pair_rows(d) && !(e && e[0] != '\0');
    if (!T.use) return T;
    // 24 rows waste less halo (256^3 147 against 155 us per iteration, 192^3 64
    // against 66), 20 rows make more CTAs of a small volume (64^3 7.2 against
    // 8.4, 96^3 10.6 against 12.3) and leave the 4-byte instantiation the
    // registers it needs (143x201x255 83 against 104, 255^3 182 against 199)
    T.aligned = aligned && d.nx % 2 == 0;
    const int rows = T.aligned && d.n >= (1LL << 20) ? 24 : 20;
    static const int r20 = resident_ctas(k_sb_pair<false, false, true, 20>, LX * 20);
    static const int r24 = resident_ctas(k_sb_pair<false, false, true, 24>, LX * 24);
    const int resident = rows == 24 ? r24 : r20;
    T.block = dim3(LX, rows, 1);
    const int gx = (d.nx + OXS - 1) / OXS, gy = (d.ny + rows - 5) / (rows - 4);
    T.zchunk = wave_zchunk((long long)gx * gy, d.nz, resident, 4, ZCHUNK);
    T.grid = dim3(gx, gy, (d.nz + T.zchunk - 1) / T.zchunk);
    T.nblocks = (long long)T.grid.x * T.grid.y * T.grid.z;
    return T;
}

int sb_pair_step(const SbPlan& T, const SbFusedArgs& a, bool aniso, const Dims& d, const StopCtl* ctl, int check,
                 double2* partials, cudaStream_t s) {
    const bool c = check != 0;
    const Kernel kern = T.block.y == 24 ? pick<24, true>(c, aniso)
                        : T.aligned     ? pick<20, true>(c, aniso)
                                        : pick<20, false>(c, aniso);
    CILREG_CUDA(launch_pdl(kern, T.grid, T.block, 0, s, a, d, T.zchunk, ctl, partials));
    return OK;
}

}  // namespace cilreg
