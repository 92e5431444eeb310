// 2D step kernels: one tile of the x-z plane per CTA.
//
// A 2D grid's volumes (5 wavefields, 8 with the P/S split, of 0.1 to a few MB each)
// live in L2, so a step costs latency, not bandwidth: two dependent launches, each a
// chain launch -> load -> stencil -> store.  The tile kernels keep that chain short.
// A CTA takes 64 columns x 4 NR rows with 256 threads (NR consecutive rows per
// thread) and makes one round trip to memory: the fields whose x or z derivative is
// taken arrive as one TMA box each (tile plus halo, zero outside the volume) under a
// single mbarrier, and meanwhile every thread loads the values of its own cells
// straight into registers.  The z stencils of a thread's rows share one column window
// read from shared memory.  Consecutive launches overlap through programmatic
// dependent launch: while the previous one drains, a kernel sets up its barrier and loads
// what was written two launches ago; what is newer it reads after griddepcontrol.wait
// (see tile2_begin).
//
// Measured on B200 against the z-marching kernels that 2D grids shared with 3D (one
// 32-cell row per CTA and TMA round trip) and their separate step-counter launch, ms per
// call: modelling 168 x 104, 240 steps 4.98 -> 1.11; RTM 680 x 380, 400 steps 10.07 -> 3.38;
// modelling 1471 x 803 (R = 6), 90 steps 4.24 -> 2.03.  RTM 4096 x 2048 438 -> 180 us per
// step, where the step streams from HBM (8.4 M cells x 108 B in 154 us without the P/S
// split: 5.9 TB/s).
//
// The arithmetic per cell is that of the 3D kernels without the y terms.
#pragma once

#include "step_kernels.cuh"

namespace ertm {

template <int R, int NR>
struct Tile2 {
    static constexpr int TZ = 4 * NR;                   // rows per CTA
    static constexpr int XB = xb_of(R);
    static constexpr int XW = TX2 + 2 * XB;             // halo box width
    static constexpr int ZH = TZ + 2 * R;               // halo box height
    static constexpr int pad(int n) { return (n + 31) / 32 * 32; }   // 128-byte TMA slots
    static constexpr int XZ = XW * ZH, X = XW * TZ, Z = TX2 * ZH;
};

// Shared by the tile kernels.  Launches alternate between two kernels, each of which writes
// what it alone loads cell by cell and the other stages: a thread's own values were last
// written two launches ago.  That launch had completed when the previous one passed its
// wait, and only then does that one let this one start.  Nothing else that changes in a pass
// is read ahead of the wait, the step index least of all: the launch before the first step
// writes it (what the host copies or clears for a pass lies a whole launch further back, or
// is no kernel, and overlaps with nothing).  So the staging warp waits and
// issues the copies first, while the others load their own values, past L1, before they
// wait.  Of it: us per step, modelling 168 x 104 4.36 -> 3.93, 680 x 380 8.20 -> 6.74;
// modelling 1471 x 803 2.10 -> 2.03 ms.  (Every warp loading before the wait: 3.81, 6.74, but
// 2.19 ms: in launches of several waves the copies are issued late.)
__device__ __forceinline__ void tile2_begin(uint64_t* bar)
{
    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        mbar_fence_init();
    }
    __syncthreads();
}
// `first`: the staging warp (0), which waits before anything else; the others, after their loads
__device__ __forceinline__ void tile2_go(bool first)
{
    if ((threadIdx.x < 32) != first) return;
    pdl_wait();
    pdl_launch();
}

// False (and the device error word set) when the tile's copies did not land in time;
// the issuing thread then waits for those that it did issue, so that the block never
// exits with a copy into its shared memory pending.
__device__ __forceinline__ bool tile2_wait(uint64_t* bar, unsigned polls, int* err, bool skipped)
{
    if (mbar_wait_bounded(bar, 0, polls)) return true;
    if (threadIdx.x == 0) {
        if (err) atomicExch(err, DEV_WAIT_TIMEOUT);
        if (!skipped) mbar_wait_bounded(bar, 0);
    }
    return false;
}

// the test hook: the first CTA does not issue the copy that holds plane skip_plane1 - 1
template <int TZ>
__device__ __forceinline__ bool tile2_skip(const KArgs& a)
{
    return a.skip_plane1 > 0 && a.skip_plane1 <= TZ && blockIdx.x == 0 && blockIdx.y == 0;
}

// ---------------------------------------------------------------------------
// Stress
// ---------------------------------------------------------------------------
template <int R, bool CPML, bool PS, int NR>
__global__ void __launch_bounds__(256, 2) k_stress2d(const __grid_constant__ StressMaps maps,
                                                     const __grid_constant__ KArgs a)
{
    using T = Tile2<R, NR>;
    constexpr int XW = T::XW, XZP = T::pad(T::XZ);
    extern __shared__ __align__(128) float sm[];
    __shared__ uint64_t bar;
    const int tx = threadIdx.x & (TX2 - 1), tr = threadIdx.x / TX2;
    const int i = blockIdx.x * TX2 + tx, kt = blockIdx.y * T::TZ, r0 = kt + tr * NR;
    const int sz = (int)a.sz;
    const bool skip = tile2_skip<T::TZ>(a);
    tile2_begin(&bar);
    tile2_go(true);
    if (threadIdx.x == 0 && !skip) {
        const int gx = (int)blockIdx.x * TX2 + XH - T::XB;
        mbar_expect_tx(&bar, 4u * 2 * T::XZ);
        tma3(sm, &maps.v[0], gx, 0, kt, &bar);          // volume row kt = grid row kt - R
        tma3(sm + XZP, &maps.v[1], gx, 0, kt, &bar);
    }
    const bool act = i < a.nx;
    float* sig[3] = {a.f[F_TXX], a.f[F_TZZ], a.f[F_TXZ]};
    float* tp = a.f[F_TP];
    const int WX = a.w[0] + a.w[1];
    const bool inx = CPML && act && (i < a.w[0] || i >= a.nx - a.w[1]);
    const int slx = i < a.w[0] ? i : i - a.nx + WX;
    float axf = 0.f, bxf = 1.f, axh = 0.f, bxh = 1.f;
    if (inx) {
        axf = __ldg(a.pa[0][0] + i); bxf = __ldg(a.pb[0][0] + i);
        axh = __ldg(a.pa[0][1] + i); bxh = __ldg(a.pb[0][1] + i);
    }
    // the thread's own cells
    float o[3][NR], otp[NR], vM[NR], vU[NR], px[2][NR], pz[2][NR];
#pragma unroll
    for (int r = 0; r < NR; r++) {
        const int k = r0 + r;
        if (!act || k >= a.nz) continue;
        const int c = k * sz + i;
#pragma unroll
        for (int q = 0; q < 3; q++) o[q][r] = __ldcg(&sig[q][c]);
        if (PS) otp[r] = __ldcg(&tp[c]);
        vM[r] = __ldg(a.M + c);
        vU[r] = __ldg(a.MU + c);
        if (CPML && inx) {
            px[0][r] = __ldcg(&a.psi[P_EXX][k * WX + slx]);
            px[1][r] = __ldcg(&a.psi[P_DXVZ][k * WX + slx]);
        }
        if (CPML && (k < a.w[4] || k >= a.nz - a.w[5])) {
            const int z = (k < a.w[4] ? k : k - a.nz + a.w[4] + a.w[5]) * a.nx + i;
            pz[0][r] = __ldcg(&a.psi[P_EZZ][z]);
            pz[1][r] = __ldcg(&a.psi[P_DZVX][z]);
        }
    }
    tile2_go(false);
    // source sample of this step, in the threads of its cell's column
    float wsrc = 0.f;
    bool src_here = i == a.ssx && r0 <= a.ssz && a.ssz < r0 + NR;
    if (src_here) {
        const int it = step_index(a);
        src_here = it >= 0 && it < a.nw;
        if (src_here) wsrc = __ldg(a.wavelet + it);
    }
    if (!tile2_wait(&bar, consumer_polls(a), a.err, skip)) return;
    if (!act || r0 >= a.nz) return;
    // tile cell (row kt + q, column i) sits at [(q + R) * XW + tx + XB]
    const float* Tx = sm + (tr * NR + R) * XW + tx + T::XB;
    const float* Tz = Tx + XZP;
    float wx[NR + 2 * R - 1], wz[NR + 2 * R - 1];   // rows 1-R.. of vx, -R.. of vz
#pragma unroll
    for (int q = 0; q < NR + 2 * R - 1; q++) {
        wx[q] = Tx[(q + 1 - R) * XW];
        wz[q] = Tz[(q - R) * XW];
    }
#pragma unroll
    for (int r = 0; r < NR; r++) {
        const int k = r0 + r;
        if (k >= a.nz) break;
        float exx = 0.f, dxvz = 0.f, ezz = 0.f, dzvx = 0.f;
#pragma unroll
        for (int n = 1; n <= R; n++) {
            exx = fmaf(a.cx[n], Tx[r * XW + n] - Tx[r * XW + 1 - n], exx);
            dxvz = fmaf(a.cx[n], Tz[r * XW + n - 1] - Tz[r * XW - n], dxvz);
            ezz = fmaf(a.cz[n], wz[r + R + n - 1] - wz[r + R - n], ezz);
            dzvx = fmaf(a.cz[n], wx[r + R - 1 + n] - wx[r + R - n], dzvx);
        }
        const int c = k * sz + i;
        if (CPML) {
            if (inx) {
                const int x = k * WX + slx;
                float p0 = fmaf(bxf, px[0][r], axf * exx);
                float p1 = fmaf(bxh, px[1][r], axh * dxvz);
                a.psi[P_EXX][x] = p0;
                a.psi[P_DXVZ][x] = p1;
                exx += p0;
                dxvz += p1;
            }
            if (k < a.w[4] || k >= a.nz - a.w[5]) {
                const int z = (k < a.w[4] ? k : k - a.nz + a.w[4] + a.w[5]) * a.nx + i;
                const float azf = __ldg(a.pa[2][0] + k), bzf = __ldg(a.pb[2][0] + k);
                const float azh = __ldg(a.pa[2][1] + k), bzh = __ldg(a.pb[2][1] + k);
                float p0 = fmaf(bzf, pz[0][r], azf * ezz);
                float p1 = fmaf(bzh, pz[1][r], azh * dzvx);
                a.psi[P_EZZ][z] = p0;
                a.psi[P_DZVX][z] = p1;
                ezz += p0;
                dzvx += p1;
            }
        }
        float g1, g2;
        damping<false>(a, CPML, i, 0, k, g1, g2);
        const float M = vM[r], U = vU[r];
        const float L = M - 2.f * U;
        const float dt = a.dt;
        const float eyy = 0.f;
        float oxx = o[0][r], ozz = o[1][r], oxz = o[2][r];
        if (src_here && k == a.ssz) {     // add_source_3D into txx, tzz
            oxx += wsrc;
            ozz += wsrc;
        }
        sig[0][c] = g1 * (g2 * oxx + dt * (M * exx + L * (eyy + ezz)));
        sig[1][c] = g1 * (g2 * ozz + dt * (M * ezz + L * (exx + eyy)));
        sig[2][c] = g1 * (g2 * oxz + dt * U * (dzvx + dxvz));
        if (PS) tp[c] = g1 * (g2 * otp[r] + dt * M * (exx + eyy + ezz));
    }
}

// ---------------------------------------------------------------------------
// Velocity
// ---------------------------------------------------------------------------
template <int R, bool CPML, int EPI, bool REC, int NR>
__global__ void __launch_bounds__(256, 2) k_velocity2d(const __grid_constant__ VelMaps maps,
                                                       const __grid_constant__ KArgs a)
{
    using T = Tile2<R, NR>;
    constexpr bool PS = EPI != EPI_NONE;
    constexpr int XW = T::XW;
    constexpr int O_XZ = T::pad(T::X), O_ZZ = O_XZ + T::pad(T::XZ), O_TP = O_ZZ + T::pad(T::Z);
    extern __shared__ __align__(128) float sm[];
    __shared__ uint64_t bar;
    const int tx = threadIdx.x & (TX2 - 1), tr = threadIdx.x / TX2;
    const int i = blockIdx.x * TX2 + tx, kt = blockIdx.y * T::TZ, r0 = kt + tr * NR;
    const int sz = (int)a.sz;
    const bool skip = tile2_skip<T::TZ>(a);
    tile2_begin(&bar);
    tile2_go(true);
    if (threadIdx.x == 0 && !skip) {
        const int gx = (int)blockIdx.x * TX2 + XH;
        mbar_expect_tx(&bar, 4u * (T::X + T::XZ + T::Z + (PS ? T::XZ : 0)));
        tma3(sm, &maps.txx, gx - T::XB, 0, kt + R, &bar);
        tma3(sm + O_XZ, &maps.txz, gx - T::XB, 0, kt, &bar);
        tma3(sm + O_ZZ, &maps.tyy, gx, 0, kt, &bar);     // 2D: the box of tzz
        if (PS) tma3(sm + O_TP, &maps.tp, gx - T::XB, 0, kt, &bar);
    }
    const bool act = i < a.nx;
    const int rec = ((REC || EPI == EPI_IMAGE) && act) ? receiver_index(a, i, 0) : -1;
    const long long nrec = (long long)a.nrx * a.nry;
    float* vx = a.f[F_VX];
    float* vz = a.f[F_VZ];
    float* vxp = a.f[F_VXP];
    float* vzp = a.f[F_VZP];
    const int WX = a.w[0] + a.w[1];
    const bool inx = CPML && act && (i < a.w[0] || i >= a.nx - a.w[1]);
    const int slx = i < a.w[0] ? i : i - a.nx + WX;
    float axf = 0.f, bxf = 1.f, axh = 0.f, bxh = 1.f;
    if (inx) {
        axf = __ldg(a.pa[0][0] + i); bxf = __ldg(a.pb[0][0] + i);
        axh = __ldg(a.pa[0][1] + i); bxh = __ldg(a.pb[0][1] + i);
    }
    float ovx[NR], ovz[NR], opx[NR], opz[NR], vb[NR], oex[NR], px[2][NR], pz[2][NR];
#pragma unroll
    for (int r = 0; r < NR; r++) {
        const int k = r0 + r;
        if (!act || k >= a.nz) continue;
        const int c = k * sz + i;
        ovx[r] = __ldcg(&vx[c]);
        ovz[r] = __ldcg(&vz[c]);
        vb[r] = __ldg(a.B + c);
        if (PS) {
            opx[r] = __ldcg(&vxp[c]);
            opz[r] = __ldcg(&vzp[c]);
        }
        if (EPI == EPI_EXCITE) oex[r] = __ldcg(&a.ex_amp2[c]);
        if (EPI == EPI_IMAGE) oex[r] = __int_as_float(__ldcg(&a.ex_time[c]));
        if (CPML && inx) {
            px[0][r] = __ldcg(&a.psi[P_DXTXX][k * WX + slx]);
            px[1][r] = __ldcg(&a.psi[P_DXTXZ][k * WX + slx]);
        }
        if (CPML && (k < a.w[4] || k >= a.nz - a.w[5])) {
            const int z = (k < a.w[4] ? k : k - a.nz + a.w[4] + a.w[5]) * a.nx + i;
            pz[0][r] = __ldcg(&a.psi[P_DZTXZ][z]);
            pz[1][r] = __ldcg(&a.psi[P_DZTZZ][z]);
        }
    }
    tile2_go(false);
    const int it = EPI != EPI_NONE || rec >= 0 ? step_index(a) : 0;
    if (!tile2_wait(&bar, consumer_polls(a), a.err, skip)) return;
    if (!act || r0 >= a.nz) return;
    const float* Txx = sm + tr * NR * XW + tx + T::XB;
    const float* Txz = sm + O_XZ + (tr * NR + R) * XW + tx + T::XB;
    const float* Tzz = sm + O_ZZ + (tr * NR + R) * TX2 + tx;
    const float* Ttp = sm + O_TP + (tr * NR + R) * XW + tx + T::XB;
    // column windows: rows -R.. of txz (D-), rows 1-R.. of tzz and tp (D+)
    float wxz[NR + 2 * R - 1], wzz[NR + 2 * R - 1], wtp[NR + 2 * R - 1];
#pragma unroll
    for (int q = 0; q < NR + 2 * R - 1; q++) {
        wxz[q] = Txz[(q - R) * XW];
        wzz[q] = Tzz[(q + 1 - R) * TX2];
        if (PS) wtp[q] = Ttp[(q + 1 - R) * XW];
    }
#pragma unroll
    for (int r = 0; r < NR; r++) {
        const int k = r0 + r;
        if (k >= a.nz) break;
        float dxtxx = 0.f, dztxz = 0.f, dxtxz = 0.f, dztzz = 0.f, dxtp = 0.f, dztp = 0.f;
#pragma unroll
        for (int n = 1; n <= R; n++) {
            dxtxx = fmaf(a.cx[n], Txx[r * XW + n - 1] - Txx[r * XW - n], dxtxx);
            dxtxz = fmaf(a.cx[n], Txz[r * XW + n] - Txz[r * XW + 1 - n], dxtxz);
            dztxz = fmaf(a.cz[n], wxz[r + R + n - 1] - wxz[r + R - n], dztxz);
            dztzz = fmaf(a.cz[n], wzz[r + R - 1 + n] - wzz[r + R - n], dztzz);
            if (PS) {
                dxtp = fmaf(a.cx[n], Ttp[r * XW + n - 1] - Ttp[r * XW - n], dxtp);
                dztp = fmaf(a.cz[n], wtp[r + R - 1 + n] - wtp[r + R - n], dztp);
            }
        }
        const int c = k * sz + i;
        if (CPML) {
            if (inx) {
                const int x = k * WX + slx;
                float p0 = fmaf(bxh, px[0][r], axh * dxtxx);
                float p1 = fmaf(bxf, px[1][r], axf * dxtxz);
                a.psi[P_DXTXX][x] = p0;
                a.psi[P_DXTXZ][x] = p1;
                dxtxx += p0;
                dxtxz += p1;
            }
            if (k < a.w[4] || k >= a.nz - a.w[5]) {
                const int z = (k < a.w[4] ? k : k - a.nz + a.w[4] + a.w[5]) * a.nx + i;
                const float azf = __ldg(a.pa[2][0] + k), bzf = __ldg(a.pb[2][0] + k);
                const float azh = __ldg(a.pa[2][1] + k), bzh = __ldg(a.pb[2][1] + k);
                float p0 = fmaf(bzf, pz[0][r], azf * dztxz);
                float p1 = fmaf(bzh, pz[1][r], azh * dztzz);
                a.psi[P_DZTXZ][z] = p0;
                a.psi[P_DZTZZ][z] = p1;
                dztxz += p0;
                dztzz += p1;
            }
        }
        float g1, g2;
        damping<false>(a, CPML, i, 0, k, g1, g2);
        const float db = a.dt * vb[r];
        const float dytxy = 0.f, dytyz = 0.f;
        float nvx = g1 * (g2 * ovx[r] + db * (dxtxx + dytxy + dztxz));
        float nvz = g1 * (g2 * ovz[r] + db * (dxtxz + dytyz + dztzz));
        float npx = 0.f, npz = 0.f;
        const float npy = 0.f;
        const float tpc = PS ? wtp[r + R - 1] : 0.f;
        if (PS) {
            // decoupled P velocity from the P-stress gradient (role of fwd_vxp_vzp_3D,
            // 3D_forward_or_back_together.cu:118); S velocity = v - v_P
            npx = g1 * (g2 * opx[r] + db * dxtp);
            npz = g1 * (g2 * opz[r] + db * dztp);
            vxp[c] = npx;
            vzp[c] = npz;
        }
        if (EPI == EPI_EXCITE) {
            // caculate_ex_amp_time_new (2D_elastic_RTM/elastic_2D_kernel_3.cu:30-48):
            // strict '>' keeps the earliest maximum of |v_P|
            float a2 = npx * npx + npy * npy + npz * npz;
            if (a2 > oex[r]) {
                a.ex_amp2[c] = a2;
                a.ex_time[c] = it;
                a.ex_v[0][c] = npx;
                a.ex_v[2][c] = npz;
                a.ex_tp[c] = tpc;
            }
        }
        if (EPI == EPI_IMAGE) {
            // imaging_inner_product_ex / imaging_correlation_ex
            // (2D_elastic_RTM/elastic_2D_kernel_3.cu:542-576) at it == excitation time
            if (__float_as_int(oex[r]) == it) {
                const float ex = a.ex_v[0][c], ey = 0.f, ez = a.ex_v[2][c];
                const float den = ex * ex + ey * ey + ez * ez;
                const float nvy = 0.f;
                if (den > 0.f) {   // a true division: 1/den overflows for denormal den
                    if (a.img[0]) a.img[0][c] = (ex * npx + ey * npy + ez * npz) / den;
                    if (a.img[1])
                        a.img[1][c] = (ex * (nvx - npx) + ey * (nvy - npy) + ez * (nvz - npz)) / den;
                }
                const float et = a.ex_tp[c];
                if (a.img[2] && et != 0.f) a.img[2][c] = tpc / et;
            }
            // receiver injection of the next (earlier) sample, reference :328
            if (rec >= 0 && k == a.rz && it > 0) {
                const float* d = a.traces + (long long)(it - 1) * nrec + rec;
                const long long cs = (long long)a.nt * nrec;
                if (a.inject_mode == 2) {
                    nvx = d[0];
                    nvz = d[2 * cs];
                } else {
                    nvx += d[0];
                    nvz += d[2 * cs];
                }
            }
        }
        vx[c] = nvx;
        vz[c] = nvz;
        if (REC && rec >= 0 && k == a.rz) {
            // write_or_add_shot_3D_surface_three, record flag 0 (:127)
            float* d = a.traces + (long long)it * nrec + rec;
            const long long cs = (long long)a.nt * nrec;
            d[0] = nvx;
            d[cs] = 0.f;
            d[2 * cs] = nvz;
        }
    }
}

// ---------------------------------------------------------------------------
// Launch helpers
// ---------------------------------------------------------------------------
template <int R, int NR>
constexpr size_t stress2d_smem()
{
    using T = Tile2<R, NR>;
    return 4 * (size_t)(2 * T::pad(T::XZ));
}
template <int R, int NR, bool PS>
constexpr size_t velocity2d_smem()
{
    using T = Tile2<R, NR>;
    return 4 * (size_t)(T::pad(T::X) + (PS ? 2 : 1) * T::pad(T::XZ) + T::pad(T::Z));
}

template <int R, int NR>
static cudaError_t launch_stress2d_nr(const Geom& g, const KArgs& a, const StressMaps& m, bool cpml, bool ps,
                                      cudaStream_t st)
{
    const dim3 grid((g.nx + TX2 - 1) / TX2, (g.nz + 4 * NR - 1) / (4 * NR));
    constexpr size_t sh = stress2d_smem<R, NR>();
    static_assert(sh <= 48 * 1024, "shared memory without opt-in");
    if (cpml)
        return ps ? launch_pdl(k_stress2d<R, true, true, NR>, grid, 256, sh, st, m, a)
                  : launch_pdl(k_stress2d<R, true, false, NR>, grid, 256, sh, st, m, a);
    return ps ? launch_pdl(k_stress2d<R, false, true, NR>, grid, 256, sh, st, m, a)
              : launch_pdl(k_stress2d<R, false, false, NR>, grid, 256, sh, st, m, a);
}

template <int R, int NR, bool C>
static cudaError_t launch_velocity2d_c(const Geom& g, const KArgs& a, const VelMaps& m, int epi, bool rec,
                                       cudaStream_t st)
{
    const dim3 grid((g.nx + TX2 - 1) / TX2, (g.nz + 4 * NR - 1) / (4 * NR));
    constexpr size_t sp = velocity2d_smem<R, NR, true>(), sn = velocity2d_smem<R, NR, false>();
    static_assert(sp <= 48 * 1024, "shared memory without opt-in");
    if (epi == EPI_EXCITE) return launch_pdl(k_velocity2d<R, C, EPI_EXCITE, false, NR>, grid, 256, sp, st, m, a);
    if (epi == EPI_IMAGE) return launch_pdl(k_velocity2d<R, C, EPI_IMAGE, false, NR>, grid, 256, sp, st, m, a);
    if (rec) return launch_pdl(k_velocity2d<R, C, EPI_NONE, true, NR>, grid, 256, sn, st, m, a);
    return launch_pdl(k_velocity2d<R, C, EPI_NONE, false, NR>, grid, 256, sn, st, m, a);
}

// rows per thread: Geom::nr2 (rows2d in setup.cu), the boxes of the maps follow it
template <int R>
cudaError_t launch_stress2d(const Geom& g, const KArgs& a, const StressMaps& m, bool cpml, bool ps, cudaStream_t st)
{
    if (g.nr2 == 4) return launch_stress2d_nr<R, 4>(g, a, m, cpml, ps, st);
    if (g.nr2 == 2) return launch_stress2d_nr<R, 2>(g, a, m, cpml, ps, st);
    return launch_stress2d_nr<R, 1>(g, a, m, cpml, ps, st);
}

template <int R>
cudaError_t launch_velocity2d(const Geom& g, const KArgs& a, const VelMaps& m, bool cpml, int epi, bool rec,
                              cudaStream_t st)
{
    if (g.nr2 == 4) return cpml ? launch_velocity2d_c<R, 4, true>(g, a, m, epi, rec, st)
                                : launch_velocity2d_c<R, 4, false>(g, a, m, epi, rec, st);
    if (g.nr2 == 2) return cpml ? launch_velocity2d_c<R, 2, true>(g, a, m, epi, rec, st)
                                : launch_velocity2d_c<R, 2, false>(g, a, m, epi, rec, st);
    return cpml ? launch_velocity2d_c<R, 1, true>(g, a, m, epi, rec, st)
                : launch_velocity2d_c<R, 1, false>(g, a, m, epi, rec, st);
}

}  // namespace ertm
