// FGP-TV iteration of a 3D volume with two voxels per thread along x and x
// neighbours by shuffles (FGP_TV_core.c:95-256): volumes below 2^23 voxels that
// do not run k_fgp_x2, of any row length.
//
// Such a volume's state stays in L2 and its iteration is a chain of a few
// planes' latencies.  k_fgp_stream takes two barriers per plane; here R2 of
// plane k and U of plane k-1 are both published before the one barrier of step
// k (U in the step before), the x neighbours of R1 and U come from the
// neighbouring thread's registers, and half the threads do the same work.  The
// sums and multiply-adds are those that the compiler forms for k_fgp_stream:
// the same bits.
//
// Time per iteration, k_fgp_stream -> this: 64^3 6.1 -> 5.0 us, 96^3 10.2 ->
// 7.6, 40x200x200 14.5 -> 11.1, 300x100x51 15.5 -> 12.6, 143x201x255 58 -> 55.
// In batches of uneven volumes the same tile gained nothing over the persistent
// schedule (12 volumes of 48 to 144: 7.6 against 7.4 ms per 100 iterations).
//
// A CTA of 16 x 16 threads holds pairs (X, X+1), X even; the pairs of threads
// 1..14 and rows 1..14 are updated.
#include <stdlib.h>

#include "fgp_tiled.cuh"
#include "pair.cuh"

namespace cilreg {

namespace {

using namespace pair;

constexpr int LX = 16, ROWS = 16;
constexpr int OXF = 2 * LX - 4, OYF = ROWS - 2;  // updated voxels of a tile
constexpr int NTF = LX * ROWS, TPF = 2 * NTF;
constexpr int ZCHUNK = 64;

struct ShflArgs {
    const float* pc[3];
    const float* po[3];
    float* pn[3];
    const float* f;
    float* u;
    float lam, multip;
    int nonneg, aniso, write_u, write_p;
};

// One tile (bx, by, bz) of one volume: the whole CTA walks its z chunk.
// CHECK: a stopping check (reads U_prev; the caller reduces pa, pb).
template <bool CHECK, bool ALIGNED>
__device__ __forceinline__ void shfl_tile(const ShflArgs& a, const Dims& d, int zc, int bx, int by, int bz, float c,
                                          float& pa_out, float& pb_out) {
    __shared__ __align__(16) float sR[2][TPF];
    __shared__ __align__(16) float sU[2][TPF];
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int nx = d.nx, ny = d.ny, nz = d.nz;
    const int X = bx * OXF - 2 + 2 * tx;  // x of the pair's first voxel
    const int y = by * OYF - 1 + ty;
    const bool upd = tx >= 1 && tx <= LX - 2 && ty >= 1 && ty <= ROWS - 2 && X < nx && y < ny;
    const bool x_first = X == 0, x_last = X + 2 == nx;
    const bool oend = !ALIGNED && X + 1 == nx;  // the pair's first voxel ends an odd row
    const int o = (ty * LX + tx) * 2;
    const int oyl = (max(ty - 1, 0) * LX + tx) * 2, oyh = (min(ty + 1, ROWS - 1) * LX + tx) * 2;
    const int col = min(max(y, 0), ny - 1) * nx + (ALIGNED ? min(max(X, 0), nx - 2) : pair_col(X, nx));
    const int dc = ALIGNED ? 1 : pair_step(X, nx);
    const int z0 = bz * zc;
    const int z1 = min(z0 + zc, nz);
    const int sxy = (int)d.sxy;
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
    const float2 cm = splat(c), mlam = splat(-a.lam), mp = splat(a.multip), zero = splat(0.f);
    float2 pa = zero, pb = zero;
    // plane k's P^{k-1}, P^{k-2} and f, loaded one plane earlier
    float2 pc[3], po[3], fv;
    auto load_plane = [&](int k) {
        const int v = min(max(k, 0), nz - 1) * sxy + col;
#pragma unroll
        for (int i = 0; i < 3; i++) {
            pc[i] = ldg2(a.pc[i] + v);
            po[i] = ldg2(a.po[i] + v);
        }
        fv = ldg2(a.f + v);
    };
    float2 rp[3] = {zero, zero, zero}, up = zero, uo = zero;  // R and U (and U_prev) of plane k-1
    load_plane(z0 - 1);
    auto step = [&](auto par, int k) {
        constexpr int P = decltype(par)::value;  // (k - z0 + 1) & 1
        // 1. R of plane k; start loading plane k+1
        float2 r[3];
#pragma unroll
        for (int i = 0; i < 3; i++) {
            r[i] = fma2(cm, sub2(pc[i], po[i]), pc[i]);
            if (k < 0) r[i] = zero;
        }
        const float2 fk = fv;
        if (k < z1) load_plane(k + 1);
        // U_prev of plane k, consumed one plane later
        float2 uon = zero;
        if (CHECK && upd && k >= z0 && k < z1) {
            const float* p = a.u + (k * sxy + col);
            uon = ALIGNED ? ld2(p) : make_float2(p[0], p[dc]);
        }
        st2(sR[P] + o, r[1]);
        __syncthreads();
        // 2. U of plane k (of planes inside the volume; others are never used)
        const float v = __shfl_up_sync(0xffffffffu, r[0].y, 1, LX);
        const float2 xl = make_float2(x_first ? 0.f : v, r[0].x);
        const float2 yl = (y == 0) ? zero : ld2(sR[P] + oyl);
        const float2 s = sub2(sub2(sub2(add2(add2(r[0], r[1]), r[2]), xl), yl), rp[2]);
        float2 u = fma2(mlam, s, fk);
        if (a.nonneg) u = make_float2(u.x < 0.f ? 0.f : u.x, u.y < 0.f ? 0.f : u.y);
        st2(sU[P] + o, u);
        // 3. P^k of plane k-1: its U was published before this step's barrier
        const int kp = k - 1;
        if (kp >= z0) {
            const float hi = __shfl_down_sync(0xffffffffu, up.x, 1, LX);
            float2 g[3] = {sub2(up, make_float2(up.y, hi)), sub2(up, ld2(sU[1 - P] + oyh)), sub2(up, u)};
            if (x_last) g[0].y = 0.f;
            if (oend) g[0].x = 0.f;
            if (y == ny - 1) g[1] = zero;
            if (kp == nz - 1) g[2] = zero;
            float2 p[3];
#pragma unroll
            for (int i = 0; i < 3; i++) p[i] = fma2(mp, g[i], rp[i]);
            if (!a.aniso) {
                const float2 den = fma2(p[2], p[2], fma2(p[0], p[0], mul2(p[1], p[1])));
                const float2 sq = make_float2((den.x > 1.f) ? rsqrtf(den.x) : 1.f,
                                              (den.y > 1.f) ? rsqrtf(den.y) : 1.f);  // within 2 ulp of 1/sqrtf
#pragma unroll
                for (int i = 0; i < 3; i++) p[i] = mul2(p[i], sq);
            } else {
#pragma unroll
                for (int i = 0; i < 3; i++) p[i] = make_float2(unit_clip(p[i].x), unit_clip(p[i].y));
            }
            if (upd) {
                const int w = kp * sxy + col;
                if (CHECK) {
                    const float2 df = sub2(up, uo);
                    const float2 dm = make_float2(df.x, oend ? 0.f : df.y), um = make_float2(up.x, oend ? 0.f : up.y);
                    pa = fma2(dm, dm, pa);
                    pb = fma2(um, um, pb);
                }
                if (a.write_u) put(a.u + w, up);
                if (a.write_p) {
#pragma unroll
                    for (int i = 0; i < 3; i++) put(a.pn[i] + w, p[i]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 3; i++) rp[i] = r[i];
        up = u;
        uo = uon;
    };
    int k = z0 - 1;
    for (; k + 1 <= z1; k += 2) {
        step(Ic<0>{}, k);
        step(Ic<1>{}, k + 1);
    }
    if (k <= z1) step(Ic<0>{}, k);
    pa_out = pa.x + pa.y;
    pb_out = pb.x + pb.y;
}

template <bool CHECK, bool ALIGNED>
__global__ void __launch_bounds__(NTF, 4) k_fgp_shfl(ShflArgs a, Dims d, int zc, float c, const float* carr,
                                                     const int* cbase, int coff, const StopCtl* ctl,
                                                     double2* partials) {
    pdl_wait();  // the previous iteration has completed (launch_pdl)
    if (pdl_many_waves()) pdl_trigger();
    if (ctl->stop) return;
    // momentum from device memory in replayed blocks
    const float cm = carr ? carr[*cbase + coff] : c;
    float pa, pb;
    shfl_tile<CHECK, ALIGNED>(a, d, zc, blockIdx.x, blockIdx.y, blockIdx.z, cm, pa, pb);
    if (!pdl_many_waves()) pdl_trigger();
    if (CHECK) block_pair_partial<NTF>(pa, pb, partials, block_slot());
}

// one iteration of every volume of a batch of one shape, a flat grid over all
// tiles (the states of the adjoint)
__global__ void __launch_bounds__(NTF, 4) k_fgp_shfl_batch(const FgpBatchVol* __restrict__ vols,
                                                           const int* __restrict__ tile_vol, int it, float c,
                                                           int nonneg, int aniso) {
    pdl_wait();  // the previous iteration has completed (launch_pdl)
    if (pdl_many_waves()) pdl_trigger();
    const FgpBatchVol& V = vols[tile_vol[blockIdx.x]];
    // the volume's pointers and extents in shared memory: in registers they spill
    __shared__ ShflArgs a;
    __shared__ Dims d;
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        for (int q = 0; q < 3; q++) {
            a.pn[q] = V.ring[it % 3][q];
            a.pc[q] = V.ring[(it + 2) % 3][q];
            a.po[q] = V.ring[(it + 1) % 3][q];
        }
        a.f = V.f;
        a.u = V.u;
        a.lam = V.lam;
        a.multip = V.multip;
        a.nonneg = nonneg;
        a.aniso = aniso;
        a.write_u = 0;
        a.write_p = 1;
        d = V.d;
    }
    __syncthreads();
    const int lt = (int)(blockIdx.x - V.tile_base), gx = V.gx, gy = V.gy;
    const int bx = lt % gx, by = (lt / gx) % gy, bz = lt / (gx * gy);
    float pa, pb;
    if (V.aligned)
        shfl_tile<false, true>(a, d, V.zc, bx, by, bz, c, pa, pb);
    else
        shfl_tile<false, false>(a, d, V.zc, bx, by, bz, c, pa, pb);
    if (!pdl_many_waves()) pdl_trigger();
}

}  // namespace

bool fgp_shfl_tile_grid(const Dims& d, int nvol, int& gx, int& gy, int& gz, int& zc) {
    if (!(d.nz > 1 && pair_rows(d))) return false;
    static const int resident = resident_ctas(k_fgp_shfl_batch, NTF);
    gx = (d.nx + OXF - 1) / OXF;
    gy = (d.ny + OYF - 1) / OYF;
    zc = wave_zchunk((long long)gx * gy * nvol, d.nz, resident, 2, ZCHUNK, 2.5);
    gz = (d.nz + zc - 1) / zc;
    return true;
}

int fgp_shfl_batch_step(const FgpBatchVol* d_vols, const int* d_tile_vol, long long ntiles, int it, float c,
                        int nonneg, int aniso, cudaStream_t s) {
    if (ntiles < 1 || ntiles > 2147483647LL) return fail(ERR_ARG, __FILE__, __LINE__, "tile count %lld", ntiles);
    CILREG_CUDA(launch_pdl(k_fgp_shfl_batch, dim3((unsigned)ntiles), dim3(LX, ROWS, 1), 0, s, d_vols, d_tile_vol, it, c,
                           nonneg, aniso));
    return OK;
}

TiledPlan fgp_shfl_plan(const Dims& d) {
    TiledPlan T;
    // CILREG_FGP_KERNEL=stream (or simple) keeps a one-voxel kernel.  From 2^23
    // voxels both are at the memory's rate (143x201x255 55 against 58 us per
    // iteration, 255^3 124 against 122).
    const char* e = getenv("CILREG_FGP_KERNEL");
    T.shfl = T.use = d.nz > 1 && pair_rows(d) && d.n < (1LL << 23) && !(e && e[0] != '\0');
    if (!T.use) return T;
    T.block = dim3(LX, ROWS, 1);
    static const int resident = resident_ctas(k_fgp_shfl<false, true>, NTF);
    const int gx = (d.nx + OXF - 1) / OXF, gy = (d.ny + OYF - 1) / OYF;
    T.zchunk = wave_zchunk((long long)gx * gy, d.nz, resident, 2, ZCHUNK, 2.5);
    T.grid = dim3(gx, gy, (d.nz + T.zchunk - 1) / T.zchunk);
    T.nblocks = (long long)T.grid.x * T.grid.y * T.grid.z;
    return T;
}

int fgp_shfl_step(const TiledPlan& T, const float* const pc[3], const float* const po[3], float* const pn[3],
                  const float* f, float* u, float lam, float c, float multip, int nonneg, int aniso, int write_u,
                  int write_p, int check, const Dims& d, const StopCtl* ctl, double2* partials, cudaStream_t s,
                  const float* carr, const int* cbase, int coff) {
    ShflArgs a;
    bool aligned = d.nx % 2 == 0 && host_aligned8(f) && host_aligned8(u);
    for (int i = 0; i < 3; i++) {
        a.pc[i] = pc[i];
        a.po[i] = po[i];
        a.pn[i] = pn[i];
        aligned = aligned && host_aligned8(pc[i]) && host_aligned8(po[i]) && host_aligned8(pn[i]);
    }
    a.f = f;
    a.u = u;
    a.lam = lam;
    a.multip = multip;
    a.nonneg = nonneg;
    a.aniso = aniso;
    a.write_u = write_u;
    a.write_p = write_p;
    const auto kern = aligned ? (check ? k_fgp_shfl<true, true> : k_fgp_shfl<false, true>)
                              : (check ? k_fgp_shfl<true, false> : k_fgp_shfl<false, false>);
    CILREG_CUDA(launch_pdl(kern, T.grid, T.block, 0, s, a, d, T.zchunk, c, carr, cbase, coff, ctl, partials));
    return OK;
}

}  // namespace cilreg
