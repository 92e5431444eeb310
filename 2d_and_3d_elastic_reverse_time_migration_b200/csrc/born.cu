// Born (linearised) modelling and its exact adjoint, 2D elastic or viscoelastic
// (generalised standard linear solid, up to 3 mechanisms), sponge boundaries.
//
// Viscoelastic stress (a = attenuation strengths tp, ts of the tau method; pi =
// rho vp^2, mu = rho vs^2 relaxed moduli; iso(m, u; e) = (m exx + (m-2u) ezz,
// m ezz + (m-2u) exx, u exz)):
//   r_l'   = ra_l r_l + rb_l iso(pi tp, mu ts; e)          (Crank-Nicolson decay)
//   sigma' = g1 (g2 sigma + dt (iso(pi kp, mu ks; e) + sum_l r_l'))
// with kp = 1 + nm tp, ks = 1 + nm ts (unrelaxed / relaxed); nm = 0 is elastic.
// This is the reference's memory-variable update (fwd_txxzzxzpp_viscoelastic_and_memory,
// 2D_elastic_RTM/viscoelastic_equation.cu:184-325, one mechanism) generalised to nm.
//
// The scattered field obeys the background scheme with secondary sources from
// relative perturbations (r_vp, r_vs, r_rho) of the migration model:
//   stress   += dt (dM e0_xx + dL e0_zz,  dM e0_zz + dL e0_xx,  dU e0_xz)
//   velocity += -dt r_rho a0
// dM = M (r_rho + 2 r_vp), dU = U (r_rho + 2 r_vs), dL = dM - 2 dU; e0 are the
// background strain rates at the start of the step and a0 = b div(sigma0) the
// background acceleration of the step.  These are the secondary sources of
// cuda_cal_dem_parameter_viscoelastic_media_new (2D_elastic_RTM/viscoelastic_equation.cu
// :2398-2505, inversion_para 2) without attenuation, and they make the Born
// operator the exact derivative of the discrete background scheme.
//
// The adjoint applies the transpose of every step in reverse order (D+ and D-
// transpose to -D- and -D+ on the zero-padded grid).  Per reverse step:
//   k_adj_vm  : velocity^T into the stress adjoint and the rho gradient from a0, then
//               (cell by cell, in registers) stress and memory variables^T with the
//               pi and mu gradients from e0 and the strain adjoint S
//   k_adj_str : velocity adjoint update with the stencils of S
// The background history (v0 at the start of each step, a0 of each step) is
// rebuilt per segment from checkpoints of the background state.
//
// Compact 2D layout: cell (i,k) at (k+R)*px + (i+BXH), zero halos; the per-shot volumes
// of a group are [type][shot][n], one 4D tensor (column, row, shot, type) to TMA.
//
// Every kernel is one tile of the x-z plane of one shot per CTA (blockIdx.z: shot), in
// the manner of step_kernels_2d.cuh: the fields that a stencil reads arrive as TMA boxes
// with halos under one mbarrier, each thread meanwhile loads the values of its own NR
// rows of one column into registers (up to 30 per cell with three mechanisms), and all
// stores come last.  A CTA makes one round trip to memory and others on the SM
// fill its wait, so a grid in L2 costs little more than the launch and a large group
// streams.  Before, each warp marched down 8-32 rows with one round trip per row.
// Measured on B200, ms per call before -> now: Born forward, 10 shots of 880 x 480, three
// mechanisms, 100 steps 34.4 -> 20.8 (5.36 TB/s of the 264 B per shot-cell and step that
// the pair of kernels cannot do without); adjoint, 8 shots of 592 x 336, elastic, 240
// steps 37.5 -> 21.2, and 16.6 with two segments less to rebuild; two CG iterations on 6
// shots of 168 x 104 54.8 -> 11.7 (12.7 before the own values were loaded ahead of the wait).
//
// Tiles start at allocated columns 64 b (cell 64 b - BXH): every row access is whole
// 128-byte lines.  Lanes on the zero halo columns load and compute and store nothing.
#include <cuda_runtime.h>

#include "born.cuh"
#include "step_kernels_2d.cuh"

namespace ertm {

namespace {

// box of a tile: columns of one shot's volume, halo rows, shot, type
__device__ __forceinline__ void tma4(float* dst, const CUtensorMap* map, int x, int z, int shot, int type,
                                     uint64_t* bar)
{
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4, %5}], [%6];\n" ::"r"(smem_u32(dst)),
        "l"(map), "r"(x), "r"(z), "r"(shot), "r"(type), "r"(smem_u32(bar))
        : "memory");
}

// The thread's place: column i (cell; the tile's columns are allocated columns 64 b ..),
// rows r0 .. r0 + NR - 1, and offsets of cell (i, r0) in the shared and per-shot volumes.
template <int R, int NR>
struct Place {
    using T = Tile2<R, NR>;
    int i, r0, kt, ax, tr;
    bool act;
    int c;                   // offset of cell (i, r0) in a volume
    long long zo;            // shot offset of the per-shot volumes
    __device__ __forceinline__ explicit Place(const BornArgs& a)
    {
        const int tx = threadIdx.x & (TX2 - 1);
        tr = threadIdx.x / TX2;
        ax = blockIdx.x * TX2;
        i = ax + tx - BXH;
        kt = blockIdx.y * T::TZ;
        r0 = kt + tr * NR;
        act = i >= 0 && i < a.nx;
        c = (int)((r0 + R) * a.px) + ax + tx;
        zo = (long long)blockIdx.z * a.ss;
    }
    // shared-memory addresses of the thread's first cell in a tile with both halos, with
    // the x halo only and with the z halo only
    __device__ __forceinline__ int xz() const { return (tr * NR + R) * T::XW + (threadIdx.x & (TX2 - 1)) + T::XB; }
    __device__ __forceinline__ int x() const { return tr * NR * T::XW + (threadIdx.x & (TX2 - 1)) + T::XB; }
    __device__ __forceinline__ int z() const { return (tr * NR + R) * TX2 + (threadIdx.x & (TX2 - 1)); }
};

// x differences at f[0] and z differences from a column window w, w[q] = row q - R (dm)
// or q + 1 - R (dp) of the thread's first row
template <int R>
__device__ __forceinline__ float dpx(const float* f, const float* cx)
{
    float s = 0.f;
#pragma unroll
    for (int n = 1; n <= R; n++) s = fmaf(cx[n], f[n] - f[1 - n], s);
    return s;
}
template <int R>
__device__ __forceinline__ float dmx(const float* f, const float* cx)
{
    float s = 0.f;
#pragma unroll
    for (int n = 1; n <= R; n++) s = fmaf(cx[n], f[n - 1] - f[-n], s);
    return s;
}
template <int R, int NR>
struct Win {
    float w[NR + 2 * R - 1];
    // f: the thread's first cell in a tile of pitch p; first: the window's first row
    __device__ __forceinline__ void load(const float* f, int p, int first)
    {
#pragma unroll
        for (int q = 0; q < NR + 2 * R - 1; q++) w[q] = f[(q + first) * p];
    }
    // forward difference at row r of a window that starts at row 1 - R
    __device__ __forceinline__ float dp(int r, const float* cz) const
    {
        float s = 0.f;
#pragma unroll
        for (int n = 1; n <= R; n++) s = fmaf(cz[n], w[r + R - 1 + n] - w[r + R - n], s);
        return s;
    }
    // backward difference at row r of a window that starts at row -R
    __device__ __forceinline__ float dm(int r, const float* cz) const
    {
        float s = 0.f;
#pragma unroll
        for (int n = 1; n <= R; n++) s = fmaf(cz[n], w[r + R + n - 1] - w[r + R - n], s);
        return s;
    }
};

// the shot's parameters: sx, sz, rx0, nrx, drx, rz
__device__ __forceinline__ int shot_par(const BornArgs& a, int q) { return __ldg(a.shot_tab + blockIdx.z * 8 + q); }

__device__ __forceinline__ int recv_of(const BornArgs& a, int i, int k)
{
    if (k != shot_par(a, 5)) return -1;
    int d = i - shot_par(a, 2);
    const int drx = shot_par(a, 4);
    if (d < 0 || d % drx) return -1;
    d /= drx;
    return d < shot_par(a, 3) ? d : -1;
}

__device__ __forceinline__ float* shot_traces(const BornArgs& a) { return a.traces + blockIdx.z * a.tstride; }

__device__ __forceinline__ void iso(float m, float u, float exx, float ezz, float exz, float* o)
{
    const float l = m - 2.f * u;
    o[0] = m * exx + l * ezz;
    o[1] = m * ezz + l * exx;
    o[2] = u * exz;
}

// ---- forward ---------------------------------------------------------------
template <int R, bool BORN, int NM, int NR>
__global__ void __launch_bounds__(256, 2) k_born_stress(const __grid_constant__ BornMaps maps,
                                                        const __grid_constant__ BornArgs a, int it)
{
    using T = Tile2<R, NR>;
    constexpr int P = T::pad(T::XZ);
    extern __shared__ __align__(128) float sm[];
    __shared__ uint64_t bar;
    const Place<R, NR> S(a);
    tile2_begin(&bar);
    tile2_go(true);
    if (threadIdx.x == 0) {
        const int gx = S.ax - T::XB, sh = blockIdx.z;
        mbar_expect_tx(&bar, 4u * (BORN ? 4 : 2) * T::XZ);
        tma4(sm, &maps.xz, gx, S.kt, sh, a.t_v0, &bar);
        tma4(sm + P, &maps.xz, gx, S.kt, sh, a.t_v0 + 1, &bar);
        if (BORN) {
            tma4(sm + 2 * P, &maps.xz, gx, S.kt, sh, a.t_v, &bar);
            tma4(sm + 3 * P, &maps.xz, gx, S.kt, sh, a.t_v + 1, &bar);
        }
    }
    const int px = (int)a.px;
    float* s0[3] = {a.s0xx + S.zo, a.s0zz + S.zo, a.s0xz + S.zo};
    float* sc[3] = {a.sxx + S.zo, a.szz + S.zo, a.sxz + S.zo};
    constexpr int ND = NM > 0 ? NM : 1;
    float o[3][NR], so[3][NR], r0v[3][ND][NR], rv[3][ND][NR];
    float g1[NR], g2[NR], pi[NR], mu[NR], dpi[NR], dmu[NR];
#pragma unroll
    for (int r = 0; r < NR; r++) {
        if (!S.act || S.r0 + r >= a.nz) continue;
        const int c = S.c + r * px;
#pragma unroll
        for (int q = 0; q < 3; q++) {
            o[q][r] = __ldcg(&s0[q][c]);
            if (BORN) so[q][r] = __ldcg(&sc[q][c]);
#pragma unroll
            for (int l = 0; l < NM; l++) {
                r0v[q][l][r] = __ldcg(&a.r0[q * 3 + l][S.zo + c]);
                if (BORN) rv[q][l][r] = __ldcg(&a.r[q * 3 + l][S.zo + c]);
            }
        }
        g1[r] = __ldg(a.g1 + c);
        g2[r] = __ldg(a.g2 + c);
        pi[r] = __ldg(a.M + c);
        mu[r] = __ldg(a.U + c);
        if (BORN) {
            dpi[r] = __ldg(a.dM + c);
            dmu[r] = __ldg(a.dU + c);
        }
    }
    const bool src_step = it >= 0 && it < a.nw;
    const bool src_col = src_step && S.i == shot_par(a, 0);
    const int srcz = shot_par(a, 1);
    tile2_go(false);
    if (!tile2_wait(&bar, kWaitPolls, a.err, false)) return;
    if (!S.act || S.r0 >= a.nz) return;
    const float* v0x = sm + S.xz();
    const float* v0z = v0x + P;
    const float* vx = v0x + 2 * P;
    const float* vz = v0x + 3 * P;
    Win<R, NR> w0x, w0z, wx, wz;      // v_x feeds forward z differences, v_z backward ones
    w0x.load(v0x, T::XW, 1 - R);
    w0z.load(v0z, T::XW, -R);
    if (BORN) {
        wx.load(vx, T::XW, 1 - R);
        wz.load(vz, T::XW, -R);
    }
    const float dt = a.dt;
#pragma unroll
    for (int r = 0; r < NR; r++) {
        const int k = S.r0 + r;
        if (k >= a.nz) break;
        const int c = S.c + r * px;
        const float e0xx = dpx<R>(v0x + r * T::XW, a.cx), e0zz = w0z.dm(r, a.cz);
        const float e0xz = w0x.dp(r, a.cz) + dmx<R>(v0z + r * T::XW, a.cx);
        float ov[3] = {o[0][r], o[1][r], o[2][r]};
        if (src_col && k == srcz) {
            // explosive source into the background
            const float w = __ldg(a.wavelet + (long long)blockIdx.z * a.wstride + it);
            ov[0] += w;
            ov[1] += w;
        }
        float E0[3], F0[3];
        iso(pi[r] * a.kp, mu[r] * a.ks, e0xx, e0zz, e0xz, E0);
        if (NM) iso(pi[r] * a.tp, mu[r] * a.ts, e0xx, e0zz, e0xz, F0);
#pragma unroll
        for (int q = 0; q < 3; q++) {
            float sum = 0.f;
#pragma unroll
            for (int l = 0; l < NM; l++) {
                const float t = a.ra[l] * r0v[q][l][r] + a.rb[l] * F0[q];
                a.r0[q * 3 + l][S.zo + c] = t;
                sum += t;
            }
            s0[q][c] = g1[r] * (g2[r] * ov[q] + dt * (E0[q] + sum));
        }
        if (BORN) {
            const float exx = dpx<R>(vx + r * T::XW, a.cx), ezz = wz.dm(r, a.cz);
            const float exz = wx.dp(r, a.cz) + dmx<R>(vz + r * T::XW, a.cx);
            float E[3], dE[3], F[3], dF[3];
            iso(pi[r] * a.kp, mu[r] * a.ks, exx, ezz, exz, E);
            // the reference's stress sources (dem_p), scaled by the GSLS strengths
            iso(dpi[r] * a.kp, dmu[r] * a.ks, e0xx, e0zz, e0xz, dE);
            if (NM) {
                iso(pi[r] * a.tp, mu[r] * a.ts, exx, ezz, exz, F);
                iso(dpi[r] * a.tp, dmu[r] * a.ts, e0xx, e0zz, e0xz, dF);
            }
#pragma unroll
            for (int q = 0; q < 3; q++) {
                float sum = 0.f;
#pragma unroll
                for (int l = 0; l < NM; l++) {
                    const float t = a.ra[l] * rv[q][l][r] + a.rb[l] * (F[q] + dF[q]);
                    a.r[q * 3 + l][S.zo + c] = t;
                    sum += t;
                }
                sc[q][c] = g1[r] * (g2[r] * so[q][r] + dt * (E[q] + dE[q] + sum));
            }
        }
    }
}

template <int R, bool BORN, bool KEEP, int NR>
__global__ void __launch_bounds__(256, 2) k_born_velocity(const __grid_constant__ BornMaps maps,
                                                          const __grid_constant__ BornArgs a, int it)
{
    using T = Tile2<R, NR>;
    constexpr int O_ZZ = T::pad(T::X), O_XZ = O_ZZ + T::pad(T::Z), FLD = O_XZ + T::pad(T::XZ);
    extern __shared__ __align__(128) float sm[];
    __shared__ uint64_t bar;
    const Place<R, NR> S(a);
    tile2_begin(&bar);
    tile2_go(true);
    if (threadIdx.x == 0) {
        const int gx = S.ax - T::XB, sh = blockIdx.z;
        mbar_expect_tx(&bar, 4u * (BORN ? 2 : 1) * (T::X + T::Z + T::XZ));
#pragma unroll
        for (int f = 0; f < (BORN ? 2 : 1); f++) {
            float* d = sm + f * FLD;
            const int t = f ? a.t_v + 2 : a.t_v0 + 2;      // sigma_xx, zz, xz
            tma4(d, &maps.x, gx, S.kt + R, sh, t, &bar);
            tma4(d + O_ZZ, &maps.z, S.ax, S.kt, sh, t + 1, &bar);
            tma4(d + O_XZ, &maps.vxz, gx, S.kt, sh, t + 2, &bar);
        }
    }
    const int px = (int)a.px;
    float* v0x = a.v0x + S.zo;
    float* v0z = a.v0z + S.zo;
    float* vx = a.vx + S.zo;
    float* vz = a.vz + S.zo;
    float ov0x[NR], ov0z[NR], ovx[NR], ovz[NR], b[NR], g1[NR], g2[NR], rr[NR];
#pragma unroll
    for (int r = 0; r < NR; r++) {
        if (!S.act || S.r0 + r >= a.nz) continue;
        const int c = S.c + r * px;
        ov0x[r] = __ldcg(&v0x[c]);
        ov0z[r] = __ldcg(&v0z[c]);
        b[r] = __ldg(a.B + c);
        g1[r] = __ldg(a.g1 + c);
        g2[r] = __ldg(a.g2 + c);
        if (BORN) {
            ovx[r] = __ldcg(&vx[c]);
            ovz[r] = __ldcg(&vz[c]);
            rr[r] = __ldg(a.rr + c);
        }
    }
    const int rz = BORN && a.traces ? shot_par(a, 5) : -1;
    tile2_go(false);
    if (!tile2_wait(&bar, kWaitPolls, a.err, false)) return;
    if (!S.act || S.r0 >= a.nz) return;
    // sigma_xz: backward z difference; sigma_zz: forward
    const float* s0xx = sm + S.x();
    const float* s0xz = sm + O_XZ + S.xz();
    Win<R, NR> w0xz, w0zz, wxz, wzz;
    w0xz.load(s0xz, T::XW, -R);
    w0zz.load(sm + O_ZZ + S.z(), TX2, 1 - R);
    if (BORN) {
        wxz.load(s0xz + FLD, T::XW, -R);
        wzz.load(sm + FLD + O_ZZ + S.z(), TX2, 1 - R);
    }
    const float dt = a.dt;
#pragma unroll
    for (int r = 0; r < NR; r++) {
        const int k = S.r0 + r;
        if (k >= a.nz) break;
        const int c = S.c + r * px;
        const float a0x = b[r] * (dmx<R>(s0xx + r * T::XW, a.cx) + w0xz.dm(r, a.cz));
        const float a0z = b[r] * (dpx<R>(s0xz + r * T::XW, a.cx) + w0zz.dp(r, a.cz));
        if (KEEP) {   // background history for the adjoint: v0 at the start of the step, a0
            const long long h = S.zo + c;
            a.kv0x[h] = ov0x[r];
            a.kv0z[h] = ov0z[r];
            a.ka0x[h] = a0x;
            a.ka0z[h] = a0z;
        }
        v0x[c] = g1[r] * (g2[r] * ov0x[r] + dt * a0x);
        v0z[c] = g1[r] * (g2[r] * ov0z[r] + dt * a0z);
        if (BORN) {
            const float ax = b[r] * (dmx<R>(s0xx + FLD + r * T::XW, a.cx) + wxz.dm(r, a.cz));
            const float az = b[r] * (dpx<R>(s0xz + FLD + r * T::XW, a.cx) + wzz.dp(r, a.cz));
            const float nvx = g1[r] * (g2[r] * ovx[r] + dt * (ax - rr[r] * a0x));
            const float nvz = g1[r] * (g2[r] * ovz[r] + dt * (az - rr[r] * a0z));
            vx[c] = nvx;
            vz[c] = nvz;
            const int rec = k == rz ? recv_of(a, S.i, k) : -1;
            if (rec >= 0) {
                const long long nrec = a.nrx, cs = (long long)a.nt * nrec;
                float* d = shot_traces(a) + (long long)it * nrec + rec;
                d[0] = nvx;
                d[cs] = 0.f;
                d[2 * cs] = nvz;
            }
        }
    }
}

// ---- adjoint ---------------------------------------------------------------
// residual sample `it` of every shot's receivers into its velocity adjoint
// (grid: receivers x, shots y)
__global__ void k_adj_inject(BornArgs a, int it)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    const int sh = blockIdx.y;
    const int* t = a.shot_tab + sh * 8;
    if (r >= t[3]) return;
    const int i = t[2] + r * t[4], rz = t[5];
    if (i < 0 || i >= a.nx || rz < 0 || rz >= a.nz) return;
    const long long c = (long long)(rz + a.R) * a.px + i + BXH + (long long)sh * a.ss;
    const long long nrec = a.nrx, cs = (long long)a.nt * nrec;
    const float* d = a.traces + sh * a.tstride + (long long)it * nrec + r;
    a.ax[c] += d[0];
    a.az[c] += d[2 * cs];
}

// velocity update^T, then stress and memory-variable update^T of one reverse step.
//
// h (the stress adjoint, already carried through g2 g1 by the previous reverse step)
// gains the velocity update's stencil transposed, applied to the products B g1 a^
// (formed in the staged tiles); rho gradient from a0.  Then, cell by cell: Q = g1 h is
// the adjoint of the stress bracket, Lambda_l = lr_l + dt Q that of r_l', P = sum_l rb_l
// Lambda_l that of f; writes the strain adjoint S = iso(pi kp, mu ks; dt Q) + iso(pi tp,
// mu ts; P) (both maps are symmetric), carries lr_l = ra_l Lambda_l and h = g2 Q,
// and accumulates the pi and mu gradients from the background strain rates.  One kernel:
// h passes between the two parts in registers (24 B per cell less, one launch less).
template <int R, int NM, int NR>
__global__ void __launch_bounds__(256, 2) k_adj_vm(const __grid_constant__ BornMaps maps,
                                                   const __grid_constant__ BornArgs a)
{
    using T = Tile2<R, NR>;
    constexpr int P = T::pad(T::XZ);
    extern __shared__ __align__(128) float sm[];
    __shared__ uint64_t bar;
    const Place<R, NR> S(a);
    tile2_begin(&bar);
    tile2_go(true);
    if (threadIdx.x == 0) {
        const int gx = S.ax - T::XB, sh = blockIdx.z;
        mbar_expect_tx(&bar, 4u * 5 * T::XZ);
        tma4(sm, &maps.xz, gx, S.kt, sh, a.t_adj, &bar);
        tma4(sm + P, &maps.xz, gx, S.kt, sh, a.t_adj + 1, &bar);
        tma4(sm + 2 * P, &maps.bg1, gx, S.kt, 0, 0, &bar);
        tma4(sm + 3 * P, &maps.hist, gx, S.kt, sh, a.t_hist, &bar);
        tma4(sm + 4 * P, &maps.hist, gx, S.kt, sh, a.t_hist + 1, &bar);
    }
    const int px = (int)a.px;
    constexpr int ND = NM > 0 ? NM : 1;
    float* h[3] = {a.hxx + S.zo, a.hzz + S.zo, a.hxz + S.zo};
    float* Sg[3] = {a.Sxx + S.zo, a.Szz + S.zo, a.Sxz + S.zo};
    float hv[3][NR], lv[3][ND][NR], gM[NR], gU[NR], gR[NR], h0x[NR], h0z[NR], vax[NR], vaz[NR];
    float g1[NR], g2[NR], pi[NR], mu[NR];
#pragma unroll
    for (int r = 0; r < NR; r++) {
        if (!S.act || S.r0 + r >= a.nz) continue;
        const int c = S.c + r * px;
        const long long cz = S.zo + c;
#pragma unroll
        for (int q = 0; q < 3; q++) {
            hv[q][r] = __ldcg(&h[q][c]);
#pragma unroll
            for (int l = 0; l < NM; l++) lv[q][l][r] = __ldcg(&a.lr[q * 3 + l][cz]);
        }
        gM[r] = __ldcg(&a.gM[cz]);
        gU[r] = __ldcg(&a.gU[cz]);
        gR[r] = __ldcg(&a.gR[cz]);
        g1[r] = __ldg(a.g1 + c);
        g2[r] = __ldg(a.g2 + c);
        pi[r] = __ldg(a.M + c);
        mu[r] = __ldg(a.U + c);
    }
    tile2_go(false);
    // the history may be the last launch's
#pragma unroll
    for (int r = 0; r < NR; r++) {
        if (!S.act || S.r0 + r >= a.nz) continue;
        h0x[r] = a.ha0x[S.zo + S.c + r * px];
        h0z[r] = a.ha0z[S.zo + S.c + r * px];
    }
    const bool landed = tile2_wait(&bar, kWaitPolls, a.err, false);
    float* fx = sm + S.xz();
    float* fz = fx + P;
#pragma unroll
    for (int r = 0; r < NR; r++) {
        vax[r] = fx[r * T::XW];
        vaz[r] = fz[r * T::XW];
    }
    __syncthreads();
    for (int q = threadIdx.x; q < T::XZ; q += 256) {      // the products B g1 a^
        const float b = sm[2 * P + q];
        sm[q] *= b;
        sm[P + q] *= b;
    }
    if (!__syncthreads_and(landed)) return;
    if (!S.act || S.r0 >= a.nz) return;
    const float* v0x = fx + 3 * P;
    const float* v0z = fx + 4 * P;
    Win<R, NR> wx, wz, w0x, w0z;
    wx.load(fx, T::XW, 1 - R);
    wz.load(fz, T::XW, -R);
    w0x.load(v0x, T::XW, 1 - R);
    w0z.load(v0z, T::XW, -R);
    const float dt = a.dt;
#pragma unroll
    for (int r = 0; r < NR; r++) {
        const int k = S.r0 + r;
        if (k >= a.nz) break;
        const int c = S.c + r * px;
        const long long cz = S.zo + c;
        const float dxx = dpx<R>(fx + r * T::XW, a.cx);
        const float dxz = wx.dp(r, a.cz) + dmx<R>(fz + r * T::XW, a.cx);
        const float dzz = wz.dm(r, a.cz);
        // rho gradient: -dt g1 (vx^ a0x + vz^ a0z)
        a.gR[cz] = gR[r] + -dt * (g1[r] * vax[r] * h0x[r] + g1[r] * vaz[r] * h0z[r]);
        const float nxx = hv[0][r] - dt * dxx, nzz = hv[1][r] - dt * dzz, nxz = hv[2][r] - dt * dxz;
        const float e0xx = dpx<R>(v0x + r * T::XW, a.cx), e0zz = w0z.dm(r, a.cz);
        const float e0xz = w0x.dp(r, a.cz) + dmx<R>(v0z + r * T::XW, a.cx);
        const float Q[3] = {g1[r] * nxx, g1[r] * nzz, g1[r] * nxz};
        float Pm[3] = {0.f, 0.f, 0.f};
#pragma unroll
        for (int q = 0; q < 3; q++)
#pragma unroll
            for (int l = 0; l < NM; l++) {
                const float lam = lv[q][l][r] + dt * Q[q];
                Pm[q] += a.rb[l] * lam;
                a.lr[q * 3 + l][cz] = a.ra[l] * lam;
            }
        const float tq0 = dt * Q[0], tq1 = dt * Q[1], tq2 = dt * Q[2];
        a.gM[cz] = gM[r] + (a.kp * (tq0 + tq1) + a.tp * (Pm[0] + Pm[1])) * (e0xx + e0zz);
        a.gU[cz] = gU[r] + (a.ks * (-2.f * tq0 * e0zz - 2.f * tq1 * e0xx + tq2 * e0xz) +
                            a.ts * (-2.f * Pm[0] * e0zz - 2.f * Pm[1] * e0xx + Pm[2] * e0xz));
        float E[3], F[3] = {0.f, 0.f, 0.f};
        iso(pi[r] * a.kp, mu[r] * a.ks, tq0, tq1, tq2, E);
        if (NM) iso(pi[r] * a.tp, mu[r] * a.ts, Pm[0], Pm[1], Pm[2], F);
#pragma unroll
        for (int q = 0; q < 3; q++) {
            Sg[q][c] = E[q] + F[q];
            h[q][c] = g2[r] * Q[q];
        }
    }
}

// velocity adjoint: a <- g2 g1 a (the velocity update^T) - D^T S (the stress
// update's stencils transposed), plus the next (earlier) step's residual
template <int R, int NR>
__global__ void __launch_bounds__(256, 2) k_adj_str(const __grid_constant__ BornMaps maps,
                                                    const __grid_constant__ BornArgs a, int it_next)
{
    using T = Tile2<R, NR>;
    constexpr int O_ZZ = T::pad(T::X), O_XZ = O_ZZ + T::pad(T::Z);
    extern __shared__ __align__(128) float sm[];
    __shared__ uint64_t bar;
    const Place<R, NR> S(a);
    tile2_begin(&bar);
    tile2_go(true);
    if (threadIdx.x == 0) {
        const int gx = S.ax - T::XB, sh = blockIdx.z;
        mbar_expect_tx(&bar, 4u * (T::X + T::Z + T::XZ));
        tma4(sm, &maps.x, gx, S.kt + R, sh, a.t_s, &bar);
        tma4(sm + O_ZZ, &maps.z, S.ax, S.kt, sh, a.t_s + 1, &bar);
        tma4(sm + O_XZ, &maps.vxz, gx, S.kt, sh, a.t_s + 2, &bar);
    }
    const int px = (int)a.px;
    float* ax = a.ax + S.zo;
    float* az = a.az + S.zo;
    float ox[NR], oz[NR], g12[NR];
#pragma unroll
    for (int r = 0; r < NR; r++) {
        if (!S.act || S.r0 + r >= a.nz) continue;
        const int c = S.c + r * px;
        ox[r] = __ldcg(&ax[c]);
        oz[r] = __ldcg(&az[c]);
        g12[r] = __ldg(a.g2 + c) * __ldg(a.g1 + c);
    }
    const int rz = it_next >= 0 ? shot_par(a, 5) : -1;
    tile2_go(false);
    if (!tile2_wait(&bar, kWaitPolls, a.err, false)) return;
    if (!S.act || S.r0 >= a.nz) return;
    const float* sxx = sm + S.x();
    const float* sxz = sm + O_XZ + S.xz();
    Win<R, NR> wxz, wzz;                  // S_xz: backward z difference; S_zz: forward
    wxz.load(sxz, T::XW, -R);
    wzz.load(sm + O_ZZ + S.z(), TX2, 1 - R);
#pragma unroll
    for (int r = 0; r < NR; r++) {
        const int k = S.r0 + r;
        if (k >= a.nz) break;
        const int c = S.c + r * px;
        const float dx = dmx<R>(sxx + r * T::XW, a.cx) + wxz.dm(r, a.cz);
        const float dz = wzz.dp(r, a.cz) + dpx<R>(sxz + r * T::XW, a.cx);
        float nx = g12[r] * ox[r] - dx;
        float nz = g12[r] * oz[r] - dz;
        const int rec = k == rz ? recv_of(a, S.i, k) : -1;
        if (rec >= 0) {
            const long long nrec = a.nrx, cs = (long long)a.nt * nrec;
            const float* d = shot_traces(a) + (long long)it_next * nrec + rec;
            nx += d[0];
            nz += d[2 * cs];
        }
        ax[c] = nx;
        az[c] = nz;
    }
}

// cell (i, k) of the small kernels below
__device__ __forceinline__ bool cell_of(const BornArgs& a, int& i, int& k, long long& c)
{
    i = blockIdx.x * blockDim.x + threadIdx.x;
    k = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= a.nx || k >= a.nz) return false;
    c = (long long)(k + a.R) * a.px + i + BXH;
    return true;
}

// gradients w.r.t. (r_vp, r_vs, r_rho) on the contiguous nz x nx grid, summed over
// the launch's shots (in shot order) and added to the outputs when `accumulate`
__global__ void k_born_final(BornArgs a, float* gvp, float* gvs, float* grho, int accumulate)
{
    int i, k;
    long long c;
    if (!cell_of(a, i, k, c)) return;
    const long long m = (long long)k * a.nx + i;
    float gp = 0.f, gu = 0.f, gr = 0.f;
    for (int sh = 0; sh < a.nshot; sh++) {
        const long long q = c + sh * a.ss;
        gp += a.gM[q];
        gu += a.gU[q];
        gr += a.gR[q];
    }
    const float ovp = accumulate ? gvp[m] : 0.f, ovs = accumulate ? gvs[m] : 0.f;
    const float orho = accumulate ? grho[m] : 0.f;
    gvp[m] = ovp + 2.f * a.M[c] * gp;
    gvs[m] = ovs + 2.f * a.U[c] * gu;
    grho[m] = orho + (a.M[c] * gp + a.U[c] * gu + gr);
}

// model products (copied from the context's padded model, plane j = 0), damping
// factors and B g1 on the compact layout
__global__ void k_born_model(BornArgs a, const float* Mc, const float* Uc, const float* Bc,
                             long long csz, const float* att_x, const float* att_z, float* M,
                             float* U, float* Bg1, float* B, float* g1, float* g2)
{
    int i, k;
    long long c;
    if (!cell_of(a, i, k, c)) return;
    const long long m = (long long)k * csz + i;
    M[c] = Mc[m];
    U[c] = Uc[m];
    B[c] = Bc[m];
    const float at = att_z[k] + att_x[i];
    const float h = at * a.dt * 0.5f;
    g1[c] = 1.f / (1.f + h);
    g2[c] = 1.f - h;
    Bg1[c] = B[c] * g1[c];
}

__global__ void k_born_pert(BornArgs a, const float* rvp, const float* rvs, const float* rrho,
                            float* dM, float* dU, float* rr)
{
    int i, k;
    long long c;
    if (!cell_of(a, i, k, c)) return;
    const long long m = (long long)k * a.nx + i;
    dM[c] = a.M[c] * (rrho[m] + 2.f * rvp[m]);
    dU[c] = a.U[c] * (rrho[m] + 2.f * rvs[m]);
    rr[c] = rrho[m];
}

dim3 born_grid(const BornArgs& a) { return dim3((a.nx + 31) / 32, (a.nz + 7) / 8); }

}  // namespace

cudaError_t born_launch_model(const BornArgs& a, const float* Mc, const float* Uc, const float* Bc,
                              long long csz, const float* att_x, const float* att_z, float* M,
                              float* U, float* Bg1, float* B, float* g1, float* g2, cudaStream_t s)
{
    k_born_model<<<born_grid(a), dim3(32, 8), 0, s>>>(a, Mc, Uc, Bc, csz, att_x, att_z, M, U, Bg1, B,
                                                      g1, g2);
    return cudaGetLastError();
}

cudaError_t born_launch_pert(const BornArgs& a, const float* rvp, const float* rvs,
                             const float* rrho, float* dM, float* dU, float* rr, cudaStream_t s)
{
    k_born_pert<<<born_grid(a), dim3(32, 8), 0, s>>>(a, rvp, rvs, rrho, dM, dU, rr);
    return cudaGetLastError();
}

namespace {
dim3 tile_grid(const BornArgs& a, int nr)
{
    return dim3((a.nx + BXH + TX2 - 1) / TX2, (a.nz + 4 * nr - 1) / (4 * nr), a.nshot);
}
template <size_t SMEM, typename... P, typename... A>
cudaError_t launch_tile(void (*K)(P...), const BornArgs& a, int nr, cudaStream_t s, const A&... args)
{
    static_assert(SMEM <= 48 * 1024, "shared memory without opt-in");
    return launch_pdl(K, tile_grid(a, nr), 256, SMEM, s, args...);
}

template <int R, int NR>
constexpr size_t xz_bytes(int n) { return 4 * (size_t)n * Tile2<R, NR>::pad(Tile2<R, NR>::XZ); }
template <int R, int NR>
constexpr size_t sig_bytes(int n)
{
    using T = Tile2<R, NR>;
    return 4 * (size_t)n * (T::pad(T::X) + T::pad(T::Z) + T::pad(T::XZ));
}

template <int R, int NM, int NR, bool BORN>
cudaError_t stress_r(const BornMaps& m, const BornArgs& a, int it, cudaStream_t s)
{
    return launch_tile<xz_bytes<R, NR>(BORN ? 4 : 2)>(k_born_stress<R, BORN, NM, NR>, a, a.nr, s, m, a, it);
}
template <int R, int NR, bool BORN, bool KEEP>
cudaError_t velocity_r(const BornMaps& m, const BornArgs& a, int it, cudaStream_t s)
{
    return launch_tile<sig_bytes<R, NR>(BORN ? 2 : 1)>(k_born_velocity<R, BORN, KEEP, NR>, a, a.nrv, s, m, a, it);
}
template <int R, int NM, bool BORN>
cudaError_t stress_nr(const BornMaps& m, const BornArgs& a, int it, cudaStream_t s)
{
    if constexpr (NM == 0)
        if (a.nr == 4) return stress_r<R, NM, 4, BORN>(m, a, it, s);
    return a.nr == 1 ? stress_r<R, NM, 1, BORN>(m, a, it, s) : stress_r<R, NM, 2, BORN>(m, a, it, s);
}
template <int R, bool BORN, bool KEEP>
cudaError_t velocity_nr(const BornMaps& m, const BornArgs& a, int it, cudaStream_t s)
{
    return a.nrv == 1   ? velocity_r<R, 1, BORN, KEEP>(m, a, it, s)
           : a.nrv == 2 ? velocity_r<R, 2, BORN, KEEP>(m, a, it, s)
                        : velocity_r<R, 4, BORN, KEEP>(m, a, it, s);
}
template <int R, int NM>
cudaError_t step_r(const BornMaps& m, const BornArgs& a, int it, bool born, bool keep, cudaStream_t s)
{
    cudaError_t e = born ? stress_nr<R, NM, true>(m, a, it, s) : stress_nr<R, NM, false>(m, a, it, s);
    if (e != cudaSuccess) return e;
    if (born) return velocity_nr<R, true, false>(m, a, it, s);
    return keep ? velocity_nr<R, false, true>(m, a, it, s) : velocity_nr<R, false, false>(m, a, it, s);
}
template <int R, int NM, int NR>
cudaError_t vm_r(const BornMaps& m, const BornArgs& a, cudaStream_t s)
{
    return launch_tile<xz_bytes<R, NR>(5)>(k_adj_vm<R, NM, NR>, a, a.nr, s, m, a);
}
template <int R, int NR>
cudaError_t str_r(const BornMaps& m, const BornArgs& a, int it, cudaStream_t s)
{
    return launch_tile<sig_bytes<R, NR>(1)>(k_adj_str<R, NR>, a, a.nrv, s, m, a, it - 1);
}
template <int R, int NM>
cudaError_t adj_r(const BornMaps& m, const BornArgs& a, int it, cudaStream_t s)
{
    cudaError_t e;
    if constexpr (NM == 0) {
        e = a.nr == 4 ? vm_r<R, NM, 4>(m, a, s) : a.nr == 2 ? vm_r<R, NM, 2>(m, a, s) : vm_r<R, NM, 1>(m, a, s);
    } else {
        e = a.nr == 2 ? vm_r<R, NM, 2>(m, a, s) : vm_r<R, NM, 1>(m, a, s);
    }
    if (e != cudaSuccess) return e;
    return a.nrv == 4 ? str_r<R, 4>(m, a, it, s) : a.nrv == 2 ? str_r<R, 2>(m, a, it, s) : str_r<R, 1>(m, a, it, s);
}
template <int R>
cudaError_t step_nm(const BornMaps& m, const BornArgs& a, int it, bool born, bool keep, cudaStream_t s)
{
    switch (a.nm) {
    case 0: return step_r<R, 0>(m, a, it, born, keep, s);
    case 1: return step_r<R, 1>(m, a, it, born, keep, s);
    case 2: return step_r<R, 2>(m, a, it, born, keep, s);
    default: return step_r<R, 3>(m, a, it, born, keep, s);
    }
}
template <int R>
cudaError_t adj_nm(const BornMaps& m, const BornArgs& a, int it, cudaStream_t s)
{
    switch (a.nm) {
    case 0: return adj_r<R, 0>(m, a, it, s);
    case 1: return adj_r<R, 1>(m, a, it, s);
    case 2: return adj_r<R, 2>(m, a, it, s);
    default: return adj_r<R, 3>(m, a, it, s);
    }
}
}  // namespace

// Rows per thread of a kernel with nm mechanisms: as many (1, 2, or 4 without memory
// variables, which take up to 24 registers a row) as still give every SM a CTA.  The
// velocity and stress^T kernels have none in any medium (10 shots of 880 x 480, three
// mechanisms: forward 22.4 -> 20.9 ms, adjoint 89 -> 84 ms with 4 rows there instead of 2).
int born_rows(int nx, int nz, int nshot, int nm)
{
    const long long cols = (nx + BXH + TX2 - 1) / TX2;
    for (int nr = nm ? 2 : 4; nr > 1; nr /= 2)
        if (cols * ((nz + 4 * nr - 1) / (4 * nr)) * nshot >= 148) return nr;
    return 1;
}

cudaError_t born_launch_step(const BornMaps& m, const BornArgs& a, int it, bool born, bool keep, cudaStream_t s)
{
    return a.R == 4 ? step_nm<4>(m, a, it, born, keep, s) : step_nm<6>(m, a, it, born, keep, s);
}

cudaError_t born_launch_adjoint_step(const BornMaps& m, const BornArgs& a, int it, cudaStream_t s)
{
    return a.R == 4 ? adj_nm<4>(m, a, it, s) : adj_nm<6>(m, a, it, s);
}

cudaError_t born_launch_inject(const BornArgs& a, int it, cudaStream_t s)
{
    if (a.nrx <= 0) return cudaSuccess;
    k_adj_inject<<<dim3((a.nrx + 127) / 128, a.nshot), 128, 0, s>>>(a, it);
    return cudaGetLastError();
}

cudaError_t born_launch_final(const BornArgs& a, float* gvp, float* gvs, float* grho, bool accumulate,
                              cudaStream_t s)
{
    k_born_final<<<born_grid(a), dim3(32, 8), 0, s>>>(a, gvp, gvs, grho, accumulate ? 1 : 0);
    return cudaGetLastError();
}

}  // namespace ertm
