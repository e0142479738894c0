// Split-Bregman TV (reference: SB_TV_core.c:38-371).
//
// Per outer iteration: two Jacobi sweeps of the (mu + 2*dim*lambda) system
// (the reference's gauss_seidel*, which read U_prev only), then shrinkage of
// grad U + B into D and the Bregman update of B.  Kernels:
//   k_sb_sweep2  both sweeps of the first outer iteration in one streaming
//                pass (sb_tiled.cu)
//   k_sb_pair    every later outer iteration of a 3D volume: as k_sb_fused,
//                two voxels per thread (sb_pair.cu)
//   k_sb_fused   every later outer iteration in one streaming pass: D and B
//                formed from U and the previous B, both sweeps, new U and B
//                written (sb_tiled.cu); D is never stored
//   k_sb_sweep   U_out = sweep(U_in, D, B, f), x2 (CILREG_SB_KERNEL=simple,
//                and volumes of 2^31 voxels or more)
//   k_sb_shrink  D, B updated in place from the new U (one voxel each): after
//                every iteration of the per-sweep path, and once at the end
//                of a warm-state (session) run of the streaming path
// The stopping check compares the two sweeps' results (SB_TV_core.c:123-134).
#include "drivers.cuh"
#include "sb_tiled.cuh"
#include "nvtx.cuh"

namespace cilreg {

namespace {

struct SbArgs {
    const float* u;   // sweep input (U_prev of the reference)
    float* un;        // sweep output
    const float* f;
    float* dd[3];
    float* bb[3];
    float lambda, mu, norm, dlam;
    int aniso, check;
};

template <bool THREE>
__global__ void __launch_bounds__(256) k_sb_sweep(SbArgs a, Dims d, int kz, const StopCtl* ctl, double2* partials) {
    if (ctl->stop) return;
    const int i = blockIdx.x * 32 + threadIdx.x;
    const int j = blockIdx.y * 8 + threadIdx.y;
    const int k0 = blockIdx.z * kz;
    float pa = 0.0f, pb = 0.0f;
    if (i < d.nx && j < d.ny) {
        const int il = nb_lo(i, d.nx), ih = nb_hi(i, d.nx), jl = nb_lo(j, d.ny), jh = nb_hi(j, d.ny);
        for (int kk = 0; kk < kz; kk++) {
            const int k = k0 + kk;
            if (k >= d.nz) break;
            const long long v = vid(d, i, j, k);
            const long long xi = vid(d, il, j, k), xo = vid(d, ih, j, k);
            const long long yi = vid(d, i, jl, k), yo = vid(d, i, jh, k);
            float sum;
            if (THREE) {
                const long long zi = vid(d, i, j, nb_lo(k, d.nz)), zo = vid(d, i, j, nb_hi(k, d.nz));
                // SB_TV_core.c:273-279
                const float dval = ldg(a.dd[0], xi) - ldg(a.dd[0], v) + ldg(a.dd[1], yi) - ldg(a.dd[1], v) +
                                   ldg(a.dd[2], zi) - ldg(a.dd[2], v);
                const float bval = -ldg(a.bb[0], xi) + ldg(a.bb[0], v) - ldg(a.bb[1], yi) + ldg(a.bb[1], v) -
                                   ldg(a.bb[2], zi) + ldg(a.bb[2], v);
                sum = dval + bval;
                sum += ldg(a.u, xo) + ldg(a.u, xi) + ldg(a.u, yo) + ldg(a.u, yi) + ldg(a.u, zo) + ldg(a.u, zi);
            } else {
                // SB_TV_core.c:166-170
                sum = ldg(a.dd[0], xi) - ldg(a.dd[0], v) + ldg(a.dd[1], yi) - ldg(a.dd[1], v) - ldg(a.bb[0], xi) +
                      ldg(a.bb[0], v) - ldg(a.bb[1], yi) + ldg(a.bb[1], v);
                sum += ldg(a.u, xo) + ldg(a.u, xi) + ldg(a.u, yo) + ldg(a.u, yi);
            }
            sum *= a.lambda;
            sum += a.mu * ldg(a.f, v);
            const float un = a.norm * sum;
            a.un[v] = un;
            if (a.check) {
                const float df = un - ldg(a.u, v);
                pa += df * df;
                pb += un * un;
            }
        }
    }
    if (a.check) block_pair_partial<256>(pa, pb, partials, block_slot());
}

template <bool THREE>
__global__ void __launch_bounds__(256) k_sb_shrink(SbArgs a, Dims d, int kz, const StopCtl* ctl) {
    if (ctl->stop) return;
    const int i = blockIdx.x * 32 + threadIdx.x;
    const int j = blockIdx.y * 8 + threadIdx.y;
    const int k0 = blockIdx.z * kz;
    if (i >= d.nx || j >= d.ny) return;
    const int ih = nb_hi(i, d.nx), jh = nb_hi(j, d.ny);
    for (int kk = 0; kk < kz; kk++) {
        const int k = k0 + kk;
        if (k >= d.nz) break;
        const long long v = vid(d, i, j, k);
        const float u = ldg(a.u, v);
        const float gx = ldg(a.u, vid(d, ih, j, k)) - u;
        const float gy = ldg(a.u, vid(d, i, jh, k)) - u;
        const float gz = THREE ? (ldg(a.u, vid(d, i, j, nb_hi(k, d.nz))) - u) : 0.0f;
        const float b1 = a.bb[0][v], b2 = a.bb[1][v], b3 = THREE ? a.bb[2][v] : 0.0f;
        const float v1 = gx + b1, v2 = gy + b2, v3 = gz + b3;
        float d1, d2, d3 = 0.0f;
        if (a.aniso) {
            // SB_TV_core.c:300-310
            const float m1 = fmaxf(fabsf(v1) - a.dlam, 0.0f);
            const float m2 = fmaxf(fabsf(v2) - a.dlam, 0.0f);
            d1 = (v1 != 0.0f) ? (v1 / fabsf(v1)) * m1 : 0.0f;
            d2 = (v2 != 0.0f) ? (v2 / fabsf(v2)) * m2 : 0.0f;
            if (THREE) {
                const float m3 = fmaxf(fabsf(v3) - a.dlam, 0.0f);
                d3 = (v3 != 0.0f) ? (v3 / fabsf(v3)) * m3 : 0.0f;
            }
        } else {
            // SB_TV_core.c:332-349
            const float den = THREE ? sqrtf(v1 * v1 + v2 * v2 + v3 * v3) : sqrtf(v1 * v1 + v2 * v2);
            const float m = fmaxf(den - a.dlam, 0.0f);
            if (den != 0.0f) {
                d1 = m * (v1 / den);
                d2 = m * (v2 / den);
                d3 = m * (v3 / den);
            } else {
                d1 = d2 = d3 = 0.0f;
            }
        }
        a.dd[0][v] = d1;
        a.dd[1][v] = d2;
        // Bregman update (SB_TV_core.c:366-368)
        a.bb[0][v] = b1 + (gx - d1);
        a.bb[1][v] = b2 + (gy - d2);
        if (THREE) {
            a.dd[2][v] = d3;
            a.bb[2][v] = b3 + (gz - d3);
        }
    }
}

}  // namespace

int sb_shrink2d(const SbSweepArgs& in, float dlam, bool aniso, const float* u, const SbWarm& warm, const Dims& d,
                const StopCtl* ctl, cudaStream_t s) {
    const Launch3 L = plan_launch(d);
    SbArgs a = {};
    for (int c = 0; c < 2; c++) {
        a.dd[c] = warm.dd[c];
        a.bb[c] = warm.bb[c];
    }
    a.u = u;
    a.lambda = in.lambda;
    a.mu = in.mu;
    a.norm = in.norm;
    a.dlam = dlam;
    a.aniso = aniso;
    a.f = in.f;
    k_sb_shrink<false><<<L.grid, L.block, 0, s>>>(a, d, L.kz, ctl);
    CILREG_CUDA(cudaGetLastError());
    note_launch();
    return OK;
}

int sb_run(const float* f, float* u_out, float mu, int iters, float epsil, int methodTV, const Dims& d,
           cudaStream_t s, float* info, SbWarm* warm) {
    CILREG_RANGE("cilreg SB-TV");
    const bool three = d.nz > 1;
    const int nc = three ? 3 : 2;
    const Launch3 L = plan_launch(d);
    if (sb_strip_applies(d)) {
        SbSweepArgs in = {};
        in.f = f;
        in.mu = 1.0f / mu;  // mu <- 1/mu, lambda = 2 mu (SB_TV_core.c:45-46)
        in.lambda = 2.0f * in.mu;
        in.norm = 1.0f / (in.mu + 4.0f * in.lambda);
        const float dlam = 1.0f / in.lambda;
        return sb_strip_run(in, dlam, methodTV == 1, u_out, iters, epsil, d, s, info, warm);
    }
    Scratch scratch(s);
    const SbPlan T = sb_sweep2_plan(d);
    bool aligned = ((uintptr_t)f | (uintptr_t)u_out) % 8 == 0;
    for (int c = 0; c < nc && warm; c++) aligned = aligned && (uintptr_t)warm->bb[c] % 8 == 0;
    const SbPlan T2 = sb_pair_plan(d, aligned);  // of the iterations k >= 1
    const long long nparts = T.use ? T.nblocks : num_blocks(L);
    IterControl ctl(s, scratch, iters, epsil, T2.use ? std::max(nparts, T2.nblocks) : nparts);
    CILREG_TRY(ctl.status());
    float* u1 = scratch.floats(d.n);
    if (!u1) return scratch.status();
    SbArgs a;
    for (int c = 0; c < 3; c++) { a.dd[c] = nullptr; a.bb[c] = nullptr; }
    for (int c = 0; c < nc; c++) {
        if (warm) {
            a.dd[c] = warm->dd[c];
            a.bb[c] = warm->bb[c];
            continue;
        }
        a.bb[c] = scratch.floats(d.n);
        if (!a.bb[c]) return scratch.status();
        CILREG_CUDA(cudaMemsetAsync(a.bb[c], 0, sizeof(float) * d.n, s));
        if (T.use) {
            a.dd[c] = a.bb[c];  // D^0 = B^0 = 0, read only by the first iteration
            continue;
        }
        a.dd[c] = scratch.floats(d.n);
        if (!a.dd[c]) return scratch.status();
        CILREG_CUDA(cudaMemsetAsync(a.dd[c], 0, sizeof(float) * d.n, s));
    }
    CILREG_CUDA(cudaMemcpyAsync(u_out, f, sizeof(float) * d.n, cudaMemcpyDeviceToDevice, s));
    // mu <- 1/mu, lambda = 2 mu (SB_TV_core.c:45-46)
    const float mu_i = 1.0f / mu;
    a.mu = mu_i;
    a.lambda = 2.0f * mu_i;
    a.norm = three ? 1.0f / (a.mu + 6.0f * a.lambda) : 1.0f / (a.mu + 4.0f * a.lambda);
    a.dlam = 1.0f / a.lambda;
    a.aniso = (methodTV == 1);
    a.f = f;
    int it = 0;
    if (T.use) {
        // Iteration 0: both sweeps with the given D^0, B^0 (k_sb_sweep2).
        // Iterations k >= 1: one pass forming D^k, B^k from U^k and B^{k-1}
        // (k_sb_fused).  U ping-pongs between u_out and u1, B between the
        // given buffers (B^0) and bb1.
        float* bufs[2] = {u_out, u1};
        float* bb1[3] = {nullptr, nullptr, nullptr};
        for (int c = 0; c < nc; c++) {
            bb1[c] = scratch.floats(d.n);
            if (!bb1[c]) return scratch.status();
        }
        float* const* bbuf[2] = {a.bb, bb1};
        SbSweepArgs w;
        for (int c = 0; c < 3; c++) {
            w.dd[c] = a.dd[c];
            w.bb[c] = a.bb[c];
        }
        w.f = f;
        w.lambda = a.lambda;
        w.mu = a.mu;
        w.norm = a.norm;
        SbFusedArgs z;
        z.f = f;
        z.lambda = a.lambda;
        z.mu = a.mu;
        z.norm = a.norm;
        z.dlam = a.dlam;
        auto later_step = [&](int check, cudaStream_t st) {
            return T2.use ? sb_pair_step(T2, z, a.aniso != 0, d, ctl.ctl(), check, ctl.partials(), st)
                          : sb_fused_step(T, z, a.aniso != 0, d, ctl.ctl(), check, ctl.partials(), st);
        };
        if (!ctl.checking() && d.n <= (1LL << 22) && iters > 1) {
            // small volume, fixed count: iteration 0 alone, iterations 1.. as
            // a replayed graph (their launches depend on the parity only)
            w.u = bufs[0];
            w.u2 = bufs[1];
            CILREG_TRY(sb_sweep2_step(T, w, d, ctl.ctl(), 0, ctl.partials(), s));
            note_launch();
            CILREG_TRY(run_replayed(iters - 1, 64, s, [&](int k, cudaStream_t st, bool) -> int {
                const int i = k + 1;
                z.u = bufs[i & 1];
                z.u2 = bufs[(i + 1) & 1];
                for (int c = 0; c < 3; c++) {
                    z.bp[c] = bbuf[(i - 1) & 1][c];
                    z.bn[c] = bbuf[i & 1][c];
                }
                CILREG_TRY(later_step(0, st));
                note_launch();
                return OK;
            }));
            it = iters;
        }
        for (; it < iters; it++) {
            const int check = ctl.is_check(it) ? 1 : 0;
            if (it == 0) {
                w.u = bufs[0];
                w.u2 = bufs[1];
                CILREG_TRY(sb_sweep2_step(T, w, d, ctl.ctl(), check, ctl.partials(), s));
            } else {
                z.u = bufs[it & 1];
                z.u2 = bufs[(it + 1) & 1];
                for (int c = 0; c < 3; c++) {
                    z.bp[c] = bbuf[(it - 1) & 1][c];
                    z.bn[c] = bbuf[it & 1][c];
                }
                CILREG_TRY(later_step(check, s));
            }
            note_launch();
            if (check) {
                CILREG_TRY(ctl.after_check(it, (it > 0 && T2.use) ? T2.nblocks : nparts));
                if (ctl.host_should_stop()) break;
            }
        }
        if (iters > 0) CILREG_TRY(launch_select_pingpong(ctl.ctl(), iters, bufs, u_out, d.n, s));
        if (warm && iters > 0) {
            // the warm state is D^n, B^n after the last iteration n - 1: bring
            // B^{n-1} (written by iteration n - 1 into bbuf[(n - 1) & 1]) into
            // warm->bb, then shrink once more from the final U, in place
            for (int c = 0; c < nc; c++) {
                float* pair[2] = {bb1[c], a.bb[c]};  // picks bbuf[last & 1]
                CILREG_TRY(launch_select_pingpong(ctl.ctl(), iters, pair, a.bb[c], d.n, s));
            }
            StopCtl* never = (StopCtl*)scratch.bytes(sizeof(StopCtl));
            if (!never) return scratch.status();
            CILREG_CUDA(cudaMemsetAsync(never, 0, sizeof(StopCtl), s));
            a.u = u_out;
            if (three) k_sb_shrink<true><<<L.grid, L.block, 0, s>>>(a, d, L.kz, never);
            else k_sb_shrink<false><<<L.grid, L.block, 0, s>>>(a, d, L.kz, never);
            CILREG_CUDA(cudaGetLastError());
            note_launch();
        }
        return ctl.finish(info);
    }
    for (; it < iters; it++) {
        const int check = ctl.is_check(it) ? 1 : 0;
        a.check = 0;
        a.u = u_out;
        a.un = u1;
        if (three) k_sb_sweep<true><<<L.grid, L.block, 0, s>>>(a, d, L.kz, ctl.ctl(), ctl.partials());
        else k_sb_sweep<false><<<L.grid, L.block, 0, s>>>(a, d, L.kz, ctl.ctl(), ctl.partials());
        CILREG_CUDA(cudaGetLastError());
        a.check = check;
        a.u = u1;
        a.un = u_out;
        if (three) k_sb_sweep<true><<<L.grid, L.block, 0, s>>>(a, d, L.kz, ctl.ctl(), ctl.partials());
        else k_sb_sweep<false><<<L.grid, L.block, 0, s>>>(a, d, L.kz, ctl.ctl(), ctl.partials());
        CILREG_CUDA(cudaGetLastError());
        a.u = u_out;
        if (three) k_sb_shrink<true><<<L.grid, L.block, 0, s>>>(a, d, L.kz, ctl.ctl());
        else k_sb_shrink<false><<<L.grid, L.block, 0, s>>>(a, d, L.kz, ctl.ctl());
        CILREG_CUDA(cudaGetLastError());
        note_launch(3);
        if (check) {
            CILREG_TRY(ctl.after_check(it, nparts));
            if (ctl.host_should_stop()) break;
        }
    }
    return ctl.finish(info);
}

}  // namespace cilreg
