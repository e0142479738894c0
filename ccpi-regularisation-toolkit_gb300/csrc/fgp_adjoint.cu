// Hand-written adjoint (vector-Jacobian product) of the unrolled FGP-TV
// iteration, with checkpointed recomputation.
//
// Forward (FGP_TV_core.c:40-269, epsil = 0, L iterations), iteration k:
//   R_k = P_{k-1} + c_k (P_{k-1} - P_{k-2})         (P_{-1} = P_{-2} = 0)
//   Z_k = f - lambda A R_k,   A R = sum_c (R_c - R_c[-e_c]),  R_c[-1] = 0
//   U_k = max(Z_k, 0) when nonneg, else Z_k
//   Q_k = R_k + m B U_k,      (B U)_c = U - U[+e_c] (0 at the last index), m = 1/(12 lambda) (1/(8 lambda) in 2D)
//   P_k = proj(Q_k)           (iso: Q / max(1, |Q|); aniso: per component)
// and the output is y = U_{L-1}.  Given ybar = dL/dy, the reverse sweep is
//   Pbar_k = (1 + c_{k+1}) Rbar_{k+1} - c_{k+2} Rbar_{k+2}
//   Qbar_k = J_proj(Q_k)^T Pbar_k
//   Zbar_k = 1[Z_k >= 0] * (m B^T Qbar_k + [k == L-1] ybar)
//   fbar  += Zbar_k
//   lambar += -<Zbar_k, A R_k> + (dm/dlambda) <Qbar_k, B U_k>
//   Rbar_k = Qbar_k - lambda A^T Zbar_k,  (A^T Z)_c = Z - Z[+e_c] (0 past the last index)
// One kernel per reverse iteration (k_adj_stream) forms Z_k, Qbar_k, Zbar_k
// and Rbar_k of every volume of a batch of equal shapes.  The forward states
// are stored every `ckpt` iterations and each segment is recomputed before its
// reverse sweep; the last segment is recomputed only, not run before as well.
// They have k_fgp_stream's roundings: the bits of the forward pass that the
// caller saw, except for images with even rows and for volumes with even rows
// whose single call runs k_fgp_x2, which round a product or two otherwise.
#include <math.h>

#include <type_traits>
#include <vector>

#include "../../include/cilreg_gb300.h"
#include "drivers.cuh"
#include "fgp_tiled.cuh"
#include "nvtx.cuh"

namespace cilreg {
namespace {

struct AdjArgs {
    const float* pm1[3];  // P_{k-1}; every array holds the volumes one after another
    const float* pm2[3];  // P_{k-2}
    const float* f;
    const float* ybar;    // only on the last iteration
    const float* rb1[3];  // Rbar_{k+1}
    const float* rb2[3];  // Rbar_{k+2}
    float* fbar;          // accumulated
    float* rb0[3];        // Rbar_k
    const float* lam;     // per volume: lambda, then m
    double2* sums;        // per CTA: <Qbar_k, B U_k> and -<Zbar_k, A R_k> over all k
    float ck, a1, a2;
    int nonneg, aniso;
};

constexpr int BX = 32, BY = 20;
constexpr int OX = BX - 4, OY = BY - 4;
constexpr int NT = BX * BY;

// The reverse iteration as a 2.5D streaming pass.  A CTA of 32 x 20 threads
// (96 registers, one per SM: backward passes 5% faster than 32 x 16; 32 x 24 at
// 80 registers and two of 32 x 16 at 64, which spill, are slower at most sizes)
// holds a tile with a two-voxel halo (R reaches one voxel down, U one up, Qbar
// one down, Zbar one up) and walks z.  Step j forms, each from what the step
// before published (two shared-memory slots, one barrier per plane) and the
// thread's registers of the planes below:
//   R of plane j;  Z, U of j-1;  Qbar of j-2;  Zbar of j-3;  Rbar of j-4.
// It reads P_{k-1}, P_{k-2}, f, Rbar_{k+1}, Rbar_{k+2}, fbar and writes Rbar_k,
// fbar: 72 bytes per voxel, against 160 and six launches when Z, A R, Qbar and
// Zbar passed through memory between four kernels and the two sums through
// reductions (4 volumes of 96^3, 60 iterations, forward and adjoint: 28 ms
// then).  Every value keeps the rounding of the separate kernels, and so do the
// sums: in FP32 over kz planes of a column (z chunks are multiples of kz), in
// FP64 beyond.
//
// IT: the type of element offsets into the batch's arrays, int below 2^31
// elements (64-bit offsets took 330 instructions per warp and plane).
template <bool THREE, typename IT>
__global__ void __launch_bounds__(NT, 1) k_adj_stream(AdjArgs a, Dims d, int zc, int nchunk, int kz) {
    pdl_wait();  // the iteration before has completed (launch_pdl)
    if (pdl_many_waves()) pdl_trigger();
    __shared__ float sR1[2][NT], sR2[2][NT], sU[2][NT], sQ1[2][NT], sQ2[2][NT], sZ[2][NT];
    const int tx = threadIdx.x, ty = threadIdx.y, o = ty * BX + tx;
    const int nx = d.nx, ny = d.ny, nz = d.nz;
    const int x = blockIdx.x * OX + tx - 2, y = blockIdx.y * OY + ty - 2;
    const int vol = blockIdx.z / nchunk;
    const int z0 = (blockIdx.z % nchunk) * zc, z1 = min(z0 + zc, nz);
    const bool in = x >= 0 && x < nx && y >= 0 && y < ny;
    const bool own = in && tx >= 2 && tx < BX - 2 && ty >= 2 && ty < BY - 2;
    const bool xl = x == nx - 1, yl = y == ny - 1;
    const int oxl = o - (tx > 0 ? 1 : 0), oxh = o + (tx < BX - 1 ? 1 : 0);
    const int oyl = o - (ty > 0 ? BX : 0), oyh = o + (ty < BY - 1 ? BX : 0);
    const float lam = a.lam[2 * vol], m = a.lam[2 * vol + 1];
    const IT base = (IT)vol * (IT)d.n + (in ? (IT)y * nx + x : 0), sxy = (IT)d.sxy;
    auto at = [&](int k) -> IT { return base + (IT)min(max(k, 0), nz - 1) * sxy; };
    constexpr int NC = THREE ? 3 : 2;
    float np[NC], npo[NC], nf, nb1[NC], nb2[NC], nfb = 0.f, nyb = 0.f;  // the next step's loads
    auto load = [&](int j) {  // R inputs of plane j, Rbar of plane j-2, fbar and ybar of plane j-3
        const IT v = at(j), w = at(j - 2);
        for (int c = 0; c < NC; c++) {
            np[c] = __ldg(a.pm1[c] + v);
            npo[c] = __ldg(a.pm2[c] + v);
            nb1[c] = __ldg(a.rb1[c] + w);
            nb2[c] = __ldg(a.rb2[c] + w);
        }
        nf = __ldg(a.f + v);
        if (own && j - 3 >= z0 && j - 3 < z1) nfb = a.fbar[at(j - 3)];
        if (a.ybar) nyb = __ldg(a.ybar + at(j - 3));
    };
    // by age: [0] plane j-1 (R) / j-1 (Z, U) ...
    float r1[3][NC] = {};                              // R of planes j-1, j-2 and j
    float f1 = 0.f;                                    // f of plane j-1
    float zv[3] = {}, ar[3] = {};                      // Z, A R of planes j-1, j-2, j-3
    float qb[3][NC] = {};                              // Qbar of planes j-2, j-3, j-4
    float zb3 = 0.f, zb4 = 0.f;                        // Zbar of planes j-3, j-4
    float r3prev = 0.f;                                // R_3 of plane j-2
    float s0 = 0.f, s1 = 0.f;
    double d0 = 0.0, d1 = 0.0;
    const int kmask = kz - 1;  // kz is a power of two
    auto clamp = [&](float z) { return (a.nonneg && z < 0.f) ? 0.f : z; };
    load(z0 - 2);
    auto step = [&](auto slot, int j) {
        constexpr int S = decltype(slot)::value, B = S ^ 1;  // slots written, read
        // R of plane j (zero outside the volume)
        float rn[NC], b1[NC], b2[NC];
        const bool rin = in && j >= 0 && j < nz;
        for (int c = 0; c < NC; c++) {
            rn[c] = rin ? __fmaf_rn(a.ck, np[c] - npo[c], np[c]) : 0.f;
            b1[c] = nb1[c];
            b2[c] = nb2[c];
        }
        const float fn = nf, fb = nfb, yb = nyb;
        if (j < z1 + 3) load(j + 1);
        sR1[S][o] = rn[0];
        sR2[S][o] = rn[1];
        // Z and U of plane j-1 (FGP_TV_core.c:220-236)
        float arn = r1[0][0] + r1[0][1];
        if (THREE) arn = arn + r1[0][NC - 1];
        arn = arn - sR1[B][oxl] - sR2[B][oyl];
        if (THREE) arn = arn - r3prev;
        const float zn = __fmaf_rn(-lam, arn, f1);
        const float un = clamp(zn);
        sU[S][o] = un;
        // Qbar of plane j-2; zv[0], ar[0] are still plane j-2's
        const int kq = j - 2;
        float qn[NC];
        {
            const float u = clamp(zv[0]);
            float bu[NC], q[NC], pb[NC];
            bu[0] = xl ? 0.f : u - sU[B][oxh];
            bu[1] = yl ? 0.f : u - sU[B][oyh];
            if (THREE) bu[NC - 1] = (kq == nz - 1) ? 0.f : u - un;
            for (int c = 0; c < NC; c++) {
                q[c] = __fmaf_rn(m, bu[c], r1[1][c]);
                pb[c] = a.a1 * b1[c] - a.a2 * b2[c];
            }
            if (!a.aniso) {
                float den = __fmaf_rn(q[0], q[0], __fmul_rn(q[1], q[1]));
                if (THREE) den = __fmaf_rn(q[NC - 1], q[NC - 1], den);
                if (den > 1.f) {
                    const float inv = 1.f / sqrtf(den);
                    float dot = q[0] * pb[0] + q[1] * pb[1];
                    if (THREE) dot += q[NC - 1] * pb[NC - 1];
                    dot *= inv;
                    for (int c = 0; c < NC; c++) qn[c] = (pb[c] - q[c] * inv * dot) * inv;
                } else {
                    for (int c = 0; c < NC; c++) qn[c] = pb[c];
                }
            } else {
                for (int c = 0; c < NC; c++) qn[c] = (fabsf(q[c]) < 1.f) ? pb[c] : 0.f;
            }
            const bool qin = in && kq >= 0 && kq < nz;
            for (int c = 0; c < NC; c++) qn[c] = qin ? qn[c] : 0.f;
            if (own && kq >= z0 && kq < z1)
                for (int c = 0; c < NC; c++) s0 += qn[c] * bu[c];
            if ((kq & kmask) == kmask || kq == nz - 1) {
                d0 += (double)s0;
                s0 = 0.f;
            }
        }
        sQ1[S][o] = qn[0];
        sQ2[S][o] = qn[1];
        // Zbar of plane j-3: qb[0] and qb[1] are still planes j-3, j-4
        const int kb = j - 3;
        float zbn = 0.f;
        if (in && kb >= 0 && kb < nz) {
            float w = (xl ? 0.f : qb[0][0]) - sQ1[B][oxl];
            w += (yl ? 0.f : qb[0][1]) - sQ2[B][oyl];
            if (THREE) w += (kb < nz - 1 ? qb[0][NC - 1] : 0.f) - qb[1][NC - 1];
            w = m * w;
            if (a.ybar) w += yb;
            zbn = (a.nonneg && zv[1] < 0.f) ? 0.f : w;
        }
        sZ[S][o] = zbn;
        if (own && kb >= z0 && kb < z1) {
            a.fbar[at(kb)] = fb + zbn;
            s1 += -zbn * ar[1];
        }
        if ((kb & kmask) == kmask || kb == nz - 1) {
            d1 += (double)s1;
            s1 = 0.f;
        }
        // Rbar of plane j-4: zb3 and qb[1] are still plane j-4's
        const int kr = j - 4;
        if (own && kr >= z0 && kr < z1) {
            const IT v = at(kr);
            a.rb0[0][v] = qb[1][0] - lam * (zb3 - sZ[B][oxh]);
            a.rb0[1][v] = qb[1][1] - lam * (zb3 - sZ[B][oyh]);
            if (THREE) a.rb0[NC - 1][v] = qb[1][NC - 1] - lam * (zb3 - zbn);
        }
        zb3 = zbn;
        r3prev = r1[0][NC - 1];
        for (int c = 0; c < NC; c++) {
            r1[1][c] = r1[0][c];
            r1[0][c] = rn[c];
            qb[1][c] = qb[0][c];
            qb[0][c] = qn[c];
        }
        f1 = fn;
        zv[1] = zv[0];
        zv[0] = zn;
        ar[1] = ar[0];
        ar[0] = arn;
        __syncthreads();
    };
    int j = z0 - 2;
    for (; j + 1 <= z1 + 3; j += 2) {
        step(std::integral_constant<int, 0>{}, j);
        step(std::integral_constant<int, 1>{}, j + 1);
    }
    if (j <= z1 + 3) step(std::integral_constant<int, 0>{}, j);
    // the volume's sums: each CTA adds to its own slot, launch after launch
    __shared__ double w0[NT / 32], w1[NT / 32];
    d0 = warp_sum(d0);
    d1 = warp_sum(d1);
    if (tx == 0) {
        w0[ty] = d0;
        w1[ty] = d1;
    }
    __syncthreads();
    if (ty == 0) {
        d0 = warp_sum(tx < NT / 32 ? w0[tx] : 0.0);
        d1 = warp_sum(tx < NT / 32 ? w1[tx] : 0.0);
        if (tx == 0) {
            double2& slot = a.sums[block_slot()];
            slot.x += d0;
            slot.y += d1;
        }
    }
}

// per volume: its CTAs' sums in a fixed order; CTA v handles volume v
__global__ void __launch_bounds__(1024) k_adj_sums(const double2* sums, long long per_vol, double2* out) {
    double s = 0.0, t = 0.0;
    for (long long p = threadIdx.x; p < per_vol; p += 1024) {
        s += sums[blockIdx.x * per_vol + p].x;
        t += sums[blockIdx.x * per_vol + p].y;
    }
    __shared__ double sa[32], sb[32];
    s = warp_sum(s);
    t = warp_sum(t);
    if ((threadIdx.x & 31) == 0) {
        sa[threadIdx.x >> 5] = s;
        sb[threadIdx.x >> 5] = t;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        s = warp_sum(sa[threadIdx.x]);
        t = warp_sum(sb[threadIdx.x]);
        if (threadIdx.x == 0) out[blockIdx.x] = make_double2(s, t);
    }
}

}  // namespace

// the vector-Jacobian products of nvol volumes of shape d that lie one after
// another in f, ybar and fbar; lams and lambar (host) hold one value per volume
int fgp_vjp_run(const float* f, const float* ybar, const float* lams, int nvol, int iters, int methodTV, int nonneg,
                int ckpt, const Dims& d, cudaStream_t s, float* fbar, double* lambar) {
    CILREG_RANGE("cilreg FGP-TV adjoint");
    if (iters < 1) return fail(ERR_ARG, __FILE__, __LINE__, "the unrolled map needs at least one iteration");
    if (ckpt < 1) ckpt = 1;
    if (ckpt > 64) return fail(ERR_ARG, __FILE__, __LINE__, "checkpoint interval %d above 64", ckpt);
    const bool three = d.nz > 1;
    const int nc = three ? 3 : 2;
    const int L = iters;
    const int nseg = (L + ckpt - 1) / ckpt, nstore = ckpt < L ? ckpt : L;
    // coefficients: iteration k forms R_k with cc[k] (cc[0] = 0), FGP_TV_core.c:138-139
    std::vector<float> cc(L + 3, 0.0f);
    {
        float tk = 1.0f, cprev = 0.0f;
        for (int k = 0; k < L + 3; k++) {
            cc[k] = cprev;
            const float tkp1 = (1.0f + sqrtf(1.0f + 4.0f * tk * tk)) * 0.5f;
            cprev = (tk - 1.0f) / tkp1;
            tk = tkp1;
        }
    }
    // tiles of the forward iteration (of fgp_shfl.cu or k_fgp_stream, the same
    // bits; every volume's one after another) and of the reverse one: 8 volumes
    // of 128^3, 60 iterations, backward 45.5 -> 42.2 ms with the former
    static const int fres = 3, ares = resident_ctas(k_adj_stream<true, int>, NT);
    int gx = 0, gy = 0, gz = 0;
    int zc = 1;
    const bool shfl = fgp_shfl_tile_grid(d, nvol, gx, gy, gz, zc);
    if (!shfl) {
        fgp_tile_grid(d, 1, gx, gy, gz);
        if (three) zc = wave_zchunk((long long)gx * gy * nvol, d.nz, fres, 2, 64);
        fgp_tile_grid(d, zc, gx, gy, gz);
    }
    const long long vtiles = (long long)gx * gy * gz;
    const int ax = (d.nx + OX - 1) / OX, ay = (d.ny + OY - 1) / OY;
    const int kz = plan_launch(d).kz;  // planes of a column summed in FP32
    const int azc = three ? (wave_zchunk((long long)ax * ay * nvol, d.nz, ares, 6, 64) + kz - 1) / kz * kz : 1;
    const int nchunk = (d.nz + azc - 1) / azc;
    if (ay > 65535 || (long long)nvol * nchunk > 65535 || vtiles * nvol > 2147483647LL)
        return fail(ERR_ARG, __FILE__, __LINE__, "%d volumes of %d x %d x %d exceed the launch grid", nvol, d.nx, d.ny,
                    d.nz);
    const dim3 agrid(ax, ay, nvol * nchunk), ablock(BX, BY, 1);
    const long long per_vol = (long long)ax * ay * nchunk;

    // one allocation for every array: checkpoints (P_{k0-1}, P_{k0-2}) of each
    // segment start k0, the forward ring, the segment's P_k, the adjoint ring
    // (an allocation each, about a hundred, cost more host time than the
    // launches, and more again from several threads)
    Scratch sc(s);
    const size_t n = (size_t)d.n * nvol, stride = (n + 63) & ~(size_t)63;
    const size_t arrays = (size_t)nc * (2 * (nseg - 1) + 3 + nstore + 3);
    float* pool = sc.floats((long long)(stride * arrays));
    const size_t ndesc = (size_t)(L + 1) * nvol;
    FgpBatchVol* d_desc = (FgpBatchVol*)sc.bytes(sizeof(FgpBatchVol) * ndesc);
    int* d_tile_vol = (int*)sc.bytes(sizeof(int) * (size_t)(vtiles * nvol));
    float* d_lam = sc.floats(2 * nvol);
    StopCtl* ctl = (StopCtl*)sc.bytes(sizeof(StopCtl));
    double2* sums = (double2*)sc.bytes(sizeof(double2) * (size_t)(per_vol * nvol + nvol));
    if (!pool || !d_desc || !d_tile_vol || !d_lam || !ctl || !sums) return sc.status();
    auto take = [&](float* out[3]) {
        for (int c = 0; c < 3; c++) {
            out[c] = c < nc ? pool : nullptr;
            if (c < nc) pool += stride;
        }
    };
    float *ring[3][3], *seg[64][3], *rbar[3][3];
    std::vector<float*> ck(6 * (nseg > 0 ? nseg : 1), nullptr);  // per segment: P_{k0-1}, P_{k0-2}
    for (int r = 0; r < 3; r++) take(ring[r]);
    for (int r = 0; r < 3; r++) take(rbar[r]);
    for (int q = 0; q < nstore; q++) take(seg[q]);
    for (int g = 1; g < nseg; g++) {
        take(&ck[6 * g]);
        take(&ck[6 * g + 3]);
    }
    const size_t nb = sizeof(float) * n;
    auto P = [&](int g, int k, int c) -> float* {  // P_k, k >= k0 - 2, while segment g is in seg
        const int k0 = g * ckpt;
        if (k >= k0) return seg[k - k0][c];
        return ck[6 * g + (k == k0 - 1 ? 0 : 3) + c];
    };
    // the first segment starts from P_{-1} = P_{-2} = 0: one array of zeros
    float* zero = sc.floats((long long)n);
    if (!zero) return sc.status();
    for (int c = 0; c < nc; c++) ck[c] = ck[3 + c] = zero;
    CILREG_CUDA(cudaMemsetAsync(zero, 0, nb, s));

    // volume descriptors: set 0 runs pass 1 on the ring, set 1 + k the
    // recomputation of iteration k into its segment's store
    std::vector<FgpBatchVol> desc(ndesc);
    std::vector<int> tile_vol((size_t)(vtiles * nvol));
    std::vector<float> lam2(2 * nvol);
    for (int v = 0; v < nvol; v++) {
        lam2[2 * v] = lams[v];
        lam2[2 * v + 1] = three ? (1.0f / (12.0f * lams[v])) : (1.0f / (8.0f * lams[v]));
        for (long long t = 0; t < vtiles; t++) tile_vol[v * vtiles + t] = v;
        for (int q = 0; q <= L; q++) {
            FgpBatchVol V = {};
            V.d = d;
            V.f = f + (size_t)v * d.n;
            V.ctl = ctl;
            V.lam = lam2[2 * v];
            V.multip = lam2[2 * v + 1];
            V.tile_base = v * vtiles;
            V.gx = gx;
            V.gy = gy;
            V.gz = gz;
            V.zc = zc;
            V.aligned = d.nx % 2 == 0 && (uintptr_t)f % 8 == 0;
            for (int c = 0; c < nc; c++) {
                const int k = q - 1, g = q > 0 ? k / ckpt : 0;
                for (int r = 0; r < 3; r++)
                    V.ring[r][c] = (q == 0 ? ring[r][c]
                                    : r == k % 3 ? seg[k - g * ckpt][c]
                                                 : P(g, r == (k + 2) % 3 ? k - 1 : k - 2, c)) +
                                   (size_t)v * d.n;
            }
            desc[(size_t)q * nvol + v] = V;
        }
    }
    CILREG_CUDA(cudaMemcpyAsync(d_desc, desc.data(), sizeof(FgpBatchVol) * ndesc, cudaMemcpyHostToDevice, s));
    CILREG_CUDA(cudaMemcpyAsync(d_tile_vol, tile_vol.data(), sizeof(int) * tile_vol.size(), cudaMemcpyHostToDevice, s));
    CILREG_CUDA(cudaMemcpyAsync(d_lam, lam2.data(), sizeof(float) * lam2.size(), cudaMemcpyHostToDevice, s));
    CILREG_TRY(launch_init_ctl(ctl, iters, s));
    CILREG_CUDA(cudaMemsetAsync(sums, 0, sizeof(double2) * (size_t)(per_vol * nvol), s));
    CILREG_CUDA(cudaMemsetAsync(fbar, 0, nb, s));
    for (int c = 0; c < nc; c++) {
        for (int r = 1; r < 3; r++) CILREG_CUDA(cudaMemsetAsync(ring[r][c], 0, nb, s));
        // Rbar_L = Rbar_{L+1} = 0
        CILREG_CUDA(cudaMemsetAsync(rbar[L % 3][c], 0, nb, s));
        CILREG_CUDA(cudaMemsetAsync(rbar[(L + 1) % 3][c], 0, nb, s));
    }
    const bool wide = d.n >= (1LL << 31), awide = (long long)d.n * nvol >= (1LL << 31);
    auto forward = [&](int set, int k) -> int {  // one production iteration of every volume
        if (shfl)
            CILREG_TRY(fgp_shfl_batch_step(d_desc + (size_t)set * nvol, d_tile_vol, vtiles * nvol, k, cc[k], nonneg == 1,
                                           methodTV != 0, s));
        else
            CILREG_TRY(fgp_batch_step(d_desc + (size_t)set * nvol, d_tile_vol, vtiles * nvol, three, wide, k, cc[k],
                                  nonneg == 1, methodTV != 0, 0, 1, 0, s));
        note_launch();
        return OK;
    };

    // pass 1: up to the last segment's start, storing (P_{k0-1}, P_{k0-2}) at each
    for (int k = 0; k <= (nseg - 1) * ckpt; k++) {
        if (k > 0 && k % ckpt == 0)
            for (int c = 0; c < nc; c++) {
                const int g = k / ckpt;
                CILREG_CUDA(cudaMemcpyAsync(ck[6 * g + c], ring[(k + 2) % 3][c], nb, cudaMemcpyDeviceToDevice, s));
                CILREG_CUDA(cudaMemcpyAsync(ck[6 * g + 3 + c], ring[(k + 1) % 3][c], nb, cudaMemcpyDeviceToDevice, s));
            }
        if (k < (nseg - 1) * ckpt) CILREG_TRY(forward(0, k));
    }
    // reverse sweep
    for (int g = nseg - 1; g >= 0; g--) {
        const int k0 = g * ckpt, k1 = (k0 + ckpt < L) ? k0 + ckpt : L;
        for (int k = k0; k < k1 - 1; k++) CILREG_TRY(forward(1 + k, k));
        for (int k = k1 - 1; k >= k0; k--) {
            AdjArgs a = {};
            for (int c = 0; c < nc; c++) {
                a.pm1[c] = P(g, k - 1, c);
                a.pm2[c] = P(g, k - 2, c);
                a.rb1[c] = rbar[(k + 1) % 3][c];
                a.rb2[c] = rbar[(k + 2) % 3][c];
                a.rb0[c] = rbar[k % 3][c];
            }
            a.f = f;
            a.ybar = (k == L - 1) ? ybar : nullptr;
            a.fbar = fbar;
            a.lam = d_lam;
            a.sums = sums;
            a.ck = cc[k];
            a.a1 = 1.0f + cc[k + 1];
            a.a2 = cc[k + 2];
            a.nonneg = (nonneg == 1);
            a.aniso = (methodTV != 0);
            auto kern = awide ? (three ? k_adj_stream<true, long long> : k_adj_stream<false, long long>)
                              : (three ? k_adj_stream<true, int> : k_adj_stream<false, int>);
            CILREG_CUDA(launch_pdl(kern, agrid, ablock, 0, s, a, d, azc, nchunk, kz));
            note_launch();
        }
    }
    double2* d_out = sums + per_vol * nvol;
    k_adj_sums<<<nvol, 1024, 0, s>>>(sums, per_vol, d_out);
    CILREG_CUDA(cudaGetLastError());
    note_launch();
    std::vector<double2> h(nvol);
    CILREG_CUDA(cudaMemcpyAsync(h.data(), d_out, sizeof(double2) * nvol, cudaMemcpyDeviceToHost, s));
    CILREG_CUDA(cudaStreamSynchronize(s));
    for (int v = 0; v < nvol && lambar; v++) {
        // d m / d lambda
        const double dm = (three ? -1.0 / 12.0 : -1.0 / 8.0) / ((double)lams[v] * lams[v]);
        lambar[v] = h[v].y + dm * h[v].x;
    }
    return OK;
}

}  // namespace cilreg

using namespace cilreg;

extern "C" int cilreg_fgp_tv_vjp_batch_dev(int nvol, const float* d_in, const float* d_ybar, float* d_inbar,
                                           double* lambar, const float* lambdaPar, int iters, int methodTV, int nonneg,
                                           int checkpoint, int dimX, int dimY, int dimZ, void* stream) {
    CILREG_TRY(check_dims(dimX, dimY, dimZ));
    if (nvol < 1) return fail(ERR_ARG, __FILE__, __LINE__, "empty batch");
    if (!d_in || !d_ybar || !d_inbar || !lambdaPar) return fail(ERR_ARG, __FILE__, __LINE__, "null pointer");
    for (int v = 0; v < nvol; v++)
        if (!(lambdaPar[v] > 0.0f)) return fail(ERR_ARG, __FILE__, __LINE__, "lambda must be positive");
    return fgp_vjp_run(d_in, d_ybar, lambdaPar, nvol, iters, methodTV, nonneg, checkpoint,
                       make_dims(dimX, dimY, dimZ < 1 ? 1 : dimZ), (cudaStream_t)stream, d_inbar, lambar);
}

extern "C" int cilreg_fgp_tv_vjp_dev(const float* d_in, const float* d_ybar, float* d_inbar, double* lambar,
                                     float lambdaPar, int iters, int methodTV, int nonneg, int checkpoint, int dimX,
                                     int dimY, int dimZ, void* stream) {
    CILREG_TRY(check_dims(dimX, dimY, dimZ));
    if (!d_in || !d_ybar || !d_inbar) return fail(ERR_ARG, __FILE__, __LINE__, "null device pointer");
    return cilreg_fgp_tv_vjp_batch_dev(1, d_in, d_ybar, d_inbar, lambar, &lambdaPar, iters, methodTV, nonneg,
                                       checkpoint, dimX, dimY, dimZ, stream);
}
