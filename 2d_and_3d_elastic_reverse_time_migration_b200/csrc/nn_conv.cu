// The U-Net's convolutions on the tensor cores: 3x3 and 2x2 transposed convolutions,
// their input gradients and their weight gradients (BF16 operands, FP32 accumulation in
// tensor memory).
//
// Operands are staged by TMA as planes of 16-byte chunks, 8 channels of one pixel per
// chunk: one 5D box (8 channels, columns, rows, chunks, image) of the NHWC view, zero
// outside the image, lands in shared memory as [chunk][row][column][16 B].  In tcgen05's
// layouts without swizzle a core matrix is 8 consecutive 16-byte rows, so the staged
// planes are read in place and from any pixel on:
//   * as a K-major operand (rows = pixels, K = channels): 128 consecutive staged pixels
//     are the M side, and a tap (ky, kx) of the 3x3 stencil is the same planes read
//     ky rows and kx pixels further.  An image row is staged with its padding column on
//     either side, so rows follow one another with a pitch of Wp pixels and 128
//     consecutive positions may run over several rows of a narrow image (the two
//     padding positions per row are computed and not stored);
//   * as an MN-major operand (rows = channels, K = pixels): the weight gradient's two
//     sides.  The planes (chunk, row) are the M side of x and the N side of dy; one MMA
//     multiplies 16 pixels of every staged row of x with those of every staged row of
//     dy, which holds the row pairs of all three ky at once (the other pairs are
//     computed and dropped: the tensor cores are far from busy), and kx is x read one
//     pixel further.
// So every pixel is staged once per tile where an im2col gather copies it nine times,
// one thread issues the copies, and the CTAs are persistent: the weights stay in shared
// memory and the copies of the next tiles run while the tensor core and the epilogue
// work on the ones before.
//
// Measured on B200 against cp.async-staged im2col tiles (and, for widths in multiples of
// 128, rows of 128 pixels), one tile per CTA: loss and gradients of a 16 x 256 x 512 batch
// 14.08 -> 3.86 ms, one 256 x 512 image forward 595 -> 274 us (bit-identical), a single
// 32 -> 48 layer on 5 x 61 x 107 with its gradients 264 -> 91 us.
//
// What bounds them: at 16-32 channels a layer moves 64-200 bytes per pixel for 5-18 kFLOP,
// the HBM side; the 16-byte rows of the boxes cost TMA about a cycle each, which is the
// other limit.
#include <algorithm>

#include "nn_common.cuh"

#include <cudaTypedefs.h>

namespace {

// ---------------------------------------------------------------------------
// Epilogues: 8 consecutive columns n0..n0+7 of output row m (n0 % 8 == 0); pre() loads
// what the epilogue needs besides the accumulators, ahead of them
// ---------------------------------------------------------------------------
struct NoPre {};

__device__ __forceinline__ uint4 pack8(const float* t)
{
    uint4 u;
    uint32_t* o = &u.x;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        __nv_bfloat162 b = __floats2bfloat162_rn(t[2 * q], t[2 * q + 1]);
        o[q] = *reinterpret_cast<uint32_t*>(&b);
    }
    return u;
}

// NHWC output (bias, optional ReLU): y[m][off + n]; N % 8 == 0
struct EpiAct {
    bf16* y;
    int cs, off, N, relu;
    const float* bias;
    typedef NoPre Pre;
    __device__ __forceinline__ Pre pre(int, int) const { return Pre(); }
    __device__ __forceinline__ void operator()(int m, int n0, const float* v, const Pre&) const
    {
        if (n0 >= N) return;
        float t[8];
#pragma unroll
        for (int q = 0; q < 8; q++) {
            t[q] = v[q] + (bias ? __ldg(bias + n0 + q) : 0.f);
            if (relu) t[q] = fmaxf(t[q], 0.f);
        }
        *reinterpret_cast<uint4*>(y + (long long)m * cs + off + n0) = pack8(t);
    }
};

// FP32 NHWC output without activation (network output)
struct EpiF32 {
    float* y;
    int cs, N, vec;          // vec: 16-byte stores are aligned
    const float* bias;
    typedef NoPre Pre;
    __device__ __forceinline__ Pre pre(int, int) const { return Pre(); }
    __device__ __forceinline__ void operator()(int m, int n0, const float* v, const Pre&) const
    {
        float* d = y + (long long)m * cs + n0;
        if (vec && n0 + 8 <= N) {
            float t[8];
#pragma unroll
            for (int q = 0; q < 8; q++) t[q] = v[q] + (bias ? __ldg(bias + n0 + q) : 0.f);
            reinterpret_cast<float4*>(d)[0] = make_float4(t[0], t[1], t[2], t[3]);
            reinterpret_cast<float4*>(d)[1] = make_float4(t[4], t[5], t[6], t[7]);
            return;
        }
#pragma unroll
        for (int q = 0; q < 8; q++) {
            if (n0 + q >= N) break;
            d[q] = v[q] + (bias ? __ldg(bias + n0 + q) : 0.f);
        }
    }
};

// input gradient: dx[m][off + n] = acc * (x[m][off + n] > 0) when mask is given
struct EpiGrad {
    bf16* dx;
    int cs, off, N;
    const bf16* mask;   // activation whose ReLU produced the layer input, same view
    typedef uint4 Pre;
    __device__ __forceinline__ Pre pre(int m, int n0) const
    {
        if (!mask || n0 >= N) return make_uint4(0, 0, 0, 0);
        return __ldg(reinterpret_cast<const uint4*>(mask + (long long)m * cs + off + n0));
    }
    __device__ __forceinline__ void operator()(int m, int n0, const float* v, const Pre& k) const
    {
        if (n0 >= N) return;
        float t[8];
        const uint32_t* w = &k.x;
#pragma unroll
        for (int q = 0; q < 8; q++) {
            t[q] = v[q];
            const uint32_t h = (q & 1) ? w[q / 2] & 0xffff0000u : w[q / 2] << 16;
            if (mask && !(__uint_as_float(h) > 0.f)) t[q] = 0.f;
        }
        *reinterpret_cast<uint4*>(dx + (long long)m * cs + off + n0) = pack8(t);
    }
};

// transposed 2x2 stride-2 convolution: column n = (a*2 + b) * C + o scatters to
// the high-resolution pixel (2i+a, 2j+b) of low-resolution row m; C % 8 == 0
struct EpiUp2 {
    bf16* y;
    int cs, off, C, lh, lw, relu;
    const float* bias;
    typedef NoPre Pre;
    __device__ __forceinline__ Pre pre(int, int) const { return Pre(); }
    __device__ __forceinline__ void operator()(int m, int n0, const float* v, const Pre&) const
    {
        if (n0 >= 4 * C) return;
        const int j = m % lw, q2 = m / lw, i = q2 % lh, nb = q2 / lh;
        const int ab = n0 / C, o = n0 - ab * C;
        float t[8];
#pragma unroll
        for (int q = 0; q < 8; q++) {
            t[q] = v[q] + (bias ? __ldg(bias + o + q) : 0.f);
            if (relu) t[q] = fmaxf(t[q], 0.f);
        }
        const long long px = (long long)(nb * 2 * lh + 2 * i + (ab >> 1)) * 2 * lw + 2 * j + (ab & 1);
        *reinterpret_cast<uint4*>(y + px * cs + off + o) = pack8(t);
    }
};

// ---------------------------------------------------------------------------
// Shared pieces
// ---------------------------------------------------------------------------
__device__ __forceinline__ void expect_tx(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(su32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive1(uint64_t* bar)
{
    asm volatile("{\n .reg .b64 st;\n mbarrier.arrive.shared::cta.b64 st, [%0];\n}\n" ::"r"(su32(bar)) : "memory");
}
__device__ __forceinline__ void tma5(void* dst, const CUtensorMap* m, int c, int x, int y, int ch, int n, uint64_t* bar)
{
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4, %5, %6}], [%7];\n" ::"r"(su32(dst)),
        "l"(m), "r"(c), "r"(x), "r"(y), "r"(ch), "r"(n), "r"(su32(bar))
        : "memory");
}
__device__ __forceinline__ void tma3w(void* dst, const CUtensorMap* m, int c, int r, int ch, uint64_t* bar)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4}], [%5];\n" ::"r"(su32(dst)),
        "l"(m), "r"(c), "r"(r), "r"(ch), "r"(su32(bar))
        : "memory");
}
__device__ __forceinline__ void tmem_ld8_nowait(uint32_t taddr, uint32_t* r)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
}
// ties the loaded registers to the wait, so that nothing reads them before it
__device__ __forceinline__ void tmem_ld_wait8(uint32_t* r)
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7])
                 :
                 : "memory");
}

constexpr int EPW = 8;                 // epilogue warps: two per quarter of the TMEM lanes
constexpr int CTHREADS = 32 * (EPW + 2);
constexpr int MAXSLOT = 16;
constexpr int SMEM_MAX = 220 * 1024;   // dynamic shared memory a CTA may take

// Tile plan of a convolution launch
struct ConvP {
    int nb, h, w;                 // output grid
    int wp, txw, ro, rows;        // staged pitch; output columns and rows of a tile; staged rows
    int halo, tx, ty, tiles;      // 1: staged rows and columns around the tile; tiles per row, row groups, tiles
    int nblk, mstep;              // 128-row MMA blocks per tile; positions from one to the next
    int C, G, nmap, taps, nch;    // channels per map, 16-channel groups per map, maps, taps and chunks per group
    int tapmajor, pair8, stream;  // K order; 8-channel taps in pairs; weights staged with each group
    int slots, nbuf, bn, tcols;
    uint32_t plane, aslot, slot;  // bytes: a chunk plane, a slot's input part, a slot
    uint32_t wtap;                // bytes of the weights of one group and tap
    uint32_t woff;                // shared-memory offset of the resident weights
};
struct ConvMaps {
    CUtensorMap x[4];             // the input (2x2 input gradient: one per output phase)
    CUtensorMap w;                // weights [N][K]: box of 8 x bn rows x 2 chunks
};

// Warps 0-7: epilogue, 8: TMA, 9: MMA.  K runs over groups of 16 channels and, inside a
// group, over its taps; with `tapmajor` over the taps and inside a tap over the groups
// (all groups of a tile staged at once): the two orders in which FP32 sums of these
// layers have always been taken, by width and channel count (see conv_plan).
template <class EP>
__global__ void __launch_bounds__(CTHREADS, 1) k_conv(const __grid_constant__ ConvMaps maps,
                                                      const __grid_constant__ ConvP p, const EP ep, int* err)
{
    extern __shared__ __align__(1024) uint8_t sm[];
    __shared__ uint64_t full[MAXSLOT], empty[MAXSLOT], tfull[2], tempty[2], wfull, done;
    __shared__ uint32_t tmem_s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = blockIdx.y * p.bn;
    const int GG = p.nmap * p.G;
    if (threadIdx.x == 0) {
        for (int q = 0; q < p.slots; q++) {
            mbar_init(&full[q], 1);
            mbar_init(&empty[q], 1);
        }
        for (int q = 0; q < 2; q++) {
            mbar_init(&tfull[q], 1);
            mbar_init(&tempty[q], EPW);
        }
        mbar_init(&wfull, 1);
        mbar_init(&done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == EPW + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(&tmem_s)),
                     "r"(p.tcols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_s;
    ertm::pdl_wait();
    ertm::pdl_launch();
    bool ok = true;
    if (warp == EPW) {
        if (lane == 0) {
            int issued = 0;
            bool wis = false;
            if (!p.stream) {          // weights of this CTA's output channels, once
                expect_tx(&wfull, (uint32_t)(GG * p.taps) * p.wtap);
                for (int gg = 0; gg < GG; gg++)
                    for (int t = 0; t < p.taps; t++) {
                        const int m = gg / p.G, g = gg - m * p.G;
                        const int kc = p.pair8 ? 2 * t : ((m + t) * p.C >> 3) + 2 * g;
                        tma3w(sm + p.woff + (uint32_t)(gg * p.taps + t) * p.wtap, &maps.w, 0, n0, kc, &wfull);
                    }
                wis = true;
            }
            for (int u = blockIdx.x; u < p.tiles && ok; u += gridDim.x) {
                const int xt = u % p.tx, q = u / p.tx, yt = q % p.ty, nb = q / p.ty;
                const int x0 = xt * p.txw - p.halo, y0 = yt * p.ro - p.halo;
                for (int gg = 0; gg < GG; gg++) {
                    const int sl = issued % p.slots, use = issued / p.slots;
                    if (use > 0 && !mbar_wait(&empty[sl], (use - 1) & 1)) {
                        ok = false;
                        break;
                    }
                    uint8_t* d = sm + (size_t)sl * p.slot;
                    const int m = gg / p.G, g = gg - m * p.G;
                    expect_tx(&full[sl], (uint32_t)p.nch * p.plane + (p.stream ? p.taps * p.wtap : 0u));
                    tma5(d, &maps.x[m], 0, x0, y0, 2 * g, nb, &full[sl]);
                    if (p.stream)
                        for (int t = 0; t < p.taps; t++)
                            tma3w(d + p.aslot + t * p.wtap, &maps.w, 0, n0, ((m + t) * p.C >> 3) + 2 * g, &full[sl]);
                    issued++;
                }
            }
            // every copy issued has landed before the block may exit
            for (int i = issued > p.slots ? issued - p.slots : 0; i < issued; i++)
                if (!mbar_wait(&full[i % p.slots], (i / p.slots) & 1)) ok = false;
            if (wis && !mbar_wait(&wfull, 0)) ok = false;
        }
        __syncwarp();
    } else if (warp == EPW + 1) {
        if (lane == 0) {
            const uint32_t idesc = idesc_bf16(p.bn);
            const uint32_t wb0 = su32(sm) + p.woff;
            int used = 0, nt = 0;
            if (!p.stream) ok = mbar_wait(&wfull, 0);
            for (int u = blockIdx.x; u < p.tiles && ok; u += gridDim.x, nt++) {
                const int buf = nt % p.nbuf, use = nt / p.nbuf;
                if (use > 0 && !mbar_wait(&tempty[buf], (use - 1) & 1)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t td = tmem + (uint32_t)(buf * p.nblk * p.bn);
                uint32_t acc = 0;
                auto mma = [&](int gg, int sl, int t) {
                    const uint32_t a0 = su32(sm) + (uint32_t)sl * p.slot;
                    const uint32_t w0 = p.stream ? a0 + p.aslot + t * p.wtap : wb0 + (uint32_t)(gg * p.taps + t) * p.wtap;
                    uint32_t shift = 0, lbo = p.plane;
                    if (p.pair8) {
                        // K = taps 2t, 2t+1 of the one chunk; the ninth has zero weights beside it
                        const int ta = 2 * t, tb = 2 * t + 1;
                        shift = (ta / 3) * p.wp + ta % 3;
                        lbo = (tb < 9 ? (tb / 3) * p.wp + tb % 3 - shift : (uint32_t)p.wp) * 16;
                    } else if (p.halo)
                        shift = (t / 3) * p.wp + t % 3;
                    const uint64_t db = sdesc(w0, p.bn * 16);
                    const uint64_t da = sdesc(a0 + shift * 16, lbo);
                    for (int b = 0; b < p.nblk; b++) umma(td + b * p.bn, da + (uint64_t)(b * p.mstep), db, idesc, acc);
                    acc = 1;
                };
                if (p.tapmajor) {
                    for (int g = 0; g < GG && ok; g++)
                        ok = mbar_wait(&full[(used + g) % p.slots], ((used + g) / p.slots) & 1);
                    if (!ok) break;
                    tc_fence_after();
                    for (int t = 0; t < p.taps; t++)
                        for (int g = 0; g < GG; g++) mma(g, (used + g) % p.slots, t);
                    for (int g = 0; g < GG; g++) umma_commit(&empty[(used + g) % p.slots]);
                    used += GG;
                } else {
                    for (int g = 0; g < GG; g++, used++) {
                        const int sl = used % p.slots;
                        if (!mbar_wait(&full[sl], (used / p.slots) & 1)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        for (int t = 0; t < p.taps; t++) mma(g, sl, t);
                        umma_commit(&empty[sl]);
                    }
                    if (!ok) break;
                }
                umma_commit(&tfull[buf]);
            }
            umma_commit(&done);       // every MMA issued has completed before TMEM is freed
            if (!mbar_wait(&done, 0)) ok = false;
        }
        __syncwarp();
    } else {
        const int quad = warp & 3, set = warp >> 2;
        int nt = 0;
        for (int u = blockIdx.x; u < p.tiles && ok; u += gridDim.x, nt++) {
            const int buf = nt % p.nbuf, use = nt / p.nbuf;
            const int xt = u % p.tx, q = u / p.tx, yt = q % p.ty, nb = q / p.ty;
            bool waited = false;
            for (int b = set; b < p.nblk; b += EPW / 4) {
                const int pos = b * p.mstep + quad * 32 + lane;
                const int r = pos / p.wp, xx = pos - r * p.wp;
                const int gx = xt * p.txw + xx, gy = yt * p.ro + r;
                const bool in = xx < p.txw && gx < p.w && r < p.ro && gy < p.h && (p.mstep == 128 || r == b);
                const int m = (nb * p.h + gy) * p.w + gx;
                const uint32_t td = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)((buf * p.nblk + b) * p.bn);
                for (int c = 0; c < p.bn; c += 32) {
                    typename EP::Pre pre[4];
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        if (in && c + 8 * k < p.bn) pre[k] = ep.pre(m, n0 + c + 8 * k);
                    if (!waited) {
                        ok = mbar_wait(&tfull[buf], use & 1);
                        waited = true;
                        tc_fence_after();
                    }
                    if (!__all_sync(0xffffffffu, ok)) {
                        ok = false;
                        break;
                    }
                    uint32_t v[4][8];
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        if (c + 8 * k < p.bn) tmem_ld8_nowait(td + c + 8 * k, v[k]);
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        if (c + 8 * k < p.bn) {
                            tmem_ld_wait8(v[k]);
                            float f[8];
#pragma unroll
                            for (int e = 0; e < 8; e++) f[e] = __uint_as_float(v[k][e]);
                            if (in) ep(m, n0 + c + 8 * k, f, pre[k]);
                        }
                }
                if (!ok) break;
            }
            if (!ok) break;
            if (!waited) {            // no block of this tile for this warp
                ok = __all_sync(0xffffffffu, mbar_wait(&tfull[buf], use & 1));
                if (!ok) break;
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive1(&tempty[buf]);
        }
    }
    if (!ok && err) atomicExch(err, NN_WAIT);
    tc_fence_before();
    __syncthreads();
    if (warp == EPW + 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(p.tcols) : "memory");
}

// ---------------------------------------------------------------------------
// Weight gradients
// ---------------------------------------------------------------------------
struct WgP {
    int nb, h, w;                 // K grid: the pixels of dy (3x3), of x (2x2)
    int tw, rr, jr;               // K tile: columns, rows of dy; staged rows of x (3x3: rr + 2)
    int tx, ty, units;
    int ci, co, CC, OC;           // channels; chunks of x and dy staged (a block of them per CTA)
    int cb;                       // channel blocks of x (grid z = cb x blocks of dy)
    int planes;                   // M side: staged planes (16 per MMA block)
    int mb, n, nkx, kgroups;      // MMA blocks, N, kx windows per CTA, groups of them
    int ksteps;
    uint32_t pitchA, pitchB, abytes, bbytes, stage;
    int stages, tcols;
    int up;                       // 2x2 transposed convolution: M = (phase, dy chunk), N = x chunks
};
struct WgMaps {
    CUtensorMap a[4], b;
};

// Partial sums of a CTA's tiles stay in TMEM (3x3: one accumulator per kx, lanes (x
// chunk, x row j, channel), columns (dy chunk, dy row r, channel)); at the end the lanes
// and columns with j - r = ky in 0..2 are the gradient of tap ky, summed over r in shared
// memory and added to dw once per CTA.  A CTA takes at most 4096 pixels per accumulator
// chain.  x and dy are read past the last column and row as zeros, so an infinite
// activation in the last column meets a zero gradient there.
__global__ void __launch_bounds__(CTHREADS, 1) k_wgrad(const __grid_constant__ WgMaps maps,
                                                       const __grid_constant__ WgP p, float* __restrict__ dw, int* err)
{
    extern __shared__ __align__(1024) uint8_t sm[];
    __shared__ uint64_t full[MAXSLOT], empty[MAXSLOT], done;
    __shared__ uint32_t tmem_s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kx0 = blockIdx.y * p.nkx;
    const int c0 = (int)(blockIdx.z % p.cb) * p.CC, o0 = (int)(blockIdx.z / p.cb) * p.OC;   // first chunks
    if (threadIdx.x == 0) {
        for (int q = 0; q < p.stages; q++) {
            mbar_init(&full[q], 1);
            mbar_init(&empty[q], 1);
        }
        mbar_init(&done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == EPW + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(&tmem_s)),
                     "r"(p.tcols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_s;
    ertm::pdl_wait();
    ertm::pdl_launch();
    bool ok = true;
    if (warp == EPW && lane == 0) {
        int i = 0;
        for (int u = blockIdx.x; u < p.units && ok; u += gridDim.x, i++) {
            const int xt = u % p.tx, q = u / p.tx, yt = q % p.ty, nb = q / p.ty;
            const int x0 = xt * p.tw, y0 = yt * p.rr;
            const int sl = i % p.stages, use = i / p.stages;
            if (use > 0 && !mbar_wait(&empty[sl], (use - 1) & 1)) {
                ok = false;
                break;
            }
            uint8_t* A = sm + (size_t)sl * p.stage;
            uint8_t* B = A + p.abytes;
            if (p.up) {
                expect_tx(&full[sl], 4u * p.OC * p.pitchA + p.bbytes);
                for (int ab = 0; ab < 4; ab++)
                    tma5(A + (uint32_t)(ab * p.OC) * p.pitchA, &maps.a[ab], 0, x0, y0, o0, nb, &full[sl]);
                tma5(B, &maps.b, 0, x0, y0, c0, nb, &full[sl]);
            } else {
                expect_tx(&full[sl], (uint32_t)(p.CC * p.jr) * p.pitchA + p.bbytes);
                tma5(A, &maps.a[0], 0, x0 - 1, y0 - 1, c0, nb, &full[sl]);
                tma5(B, &maps.b, 0, x0, y0, o0, nb, &full[sl]);
            }
        }
        for (int k = i > p.stages ? i - p.stages : 0; k < i; k++)
            if (!mbar_wait(&full[k % p.stages], (k / p.stages) & 1)) ok = false;
    } else if (warp == EPW + 1 && lane == 0) {
        const uint32_t idesc = idesc_bf16(p.n) | 1u << 15 | 1u << 16;   // both operands MN-major
        int i = 0;
        for (int u = blockIdx.x; u < p.units; u += gridDim.x, i++) {
            const int sl = i % p.stages;
            if (!mbar_wait(&full[sl], (i / p.stages) & 1)) {
                ok = false;
                break;
            }
            tc_fence_after();
            const uint32_t A = su32(sm) + (uint32_t)sl * p.stage, B = A + p.abytes;
            for (int s = 0; s < p.ksteps; s++) {
                const uint64_t db = sdesc(B + s * 256, 128, p.pitchB);
                for (int k = 0; k < p.nkx; k++)
                    for (int b = 0; b < p.mb; b++) {
                        const uint64_t da = sdesc(A + (uint32_t)b * 16 * p.pitchA + (kx0 + k + 16 * s) * 16, 128, p.pitchA);
                        umma(tmem + (uint32_t)((k * p.mb + b) * p.n), da, db, idesc, (i > 0 || s > 0) ? 1u : 0u);
                    }
            }
            umma_commit(&empty[sl]);
        }
        umma_commit(&done);
        if (!mbar_wait(&done, 0)) ok = false;
    }
    // TMEM loads are warp-collective and shared memory is reused: the decision is the block's
    const bool all_ok = __syncthreads_and(ok ? 1 : 0) != 0;
    tc_fence_after();
    if (all_ok) {
        const int quad = warp & 3, set = warp >> 2;
        const bool epi = warp < EPW;
        const int row = quad * 32 + lane;
        float* acc = reinterpret_cast<float*>(sm);
        const int cw = p.CC * 8, ow = p.OC * 8, na = ow * 9 * cw;
        const bool direct = p.up || p.rr == 1;
        if (!direct) {
            for (int q = threadIdx.x; q < na; q += CTHREADS) acc[q] = 0.f;
            __syncthreads();
        }
        for (int rs = 0; rs < (direct ? 1 : p.rr); rs++) {
            // in shared memory one dy row r at a time: then j - r = ky names every sum once
            if (epi)
                for (int t = set; t < p.nkx * p.mb; t += EPW / 4) {
                    const int k = t / p.mb, b = t - k * p.mb, m8 = b * 16 + row / 8;
                    const uint32_t td = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(t * p.n);
                    const int kx = kx0 + k;
                    for (int n8 = 0; n8 < p.n / 8; n8++) {
                        if (!p.up && !direct && n8 % p.rr != rs) continue;
                        float v[8];
                        tmem_ld8(td + n8 * 8, v);
                        if (m8 >= p.planes) continue;
                        if (p.up) {
                            const int ab = m8 / p.OC, o = (o0 + m8 - ab * p.OC) * 8 + row % 8, c = (c0 + n8) * 8;
                            if (o >= p.co || c >= p.ci) continue;
                            float* d = dw + (long long)(ab * p.co + o) * p.ci + c;
#pragma unroll
                            for (int q = 0; q < 8; q++) atomicAdd(d + q, v[q]);
                            continue;
                        }
                        const int cc = m8 / p.jr, j = m8 - cc * p.jr, oc = n8 / p.rr, r = n8 - oc * p.rr;
                        const int ky = j - r;
                        if (ky < 0 || ky > 2 || kx > 2) continue;
                        const int tap = ky * 3 + kx;
                        if (direct) {
                            const int c = (c0 + cc) * 8 + row % 8, o = (o0 + oc) * 8;
                            if (c >= p.ci || o >= p.co) continue;
#pragma unroll
                            for (int q = 0; q < 8; q++) atomicAdd(dw + ((long long)(o + q) * 9 + tap) * p.ci + c, v[q]);
                        } else {
#pragma unroll
                            for (int q = 0; q < 8; q++) acc[((oc * 8 + q) * 9 + tap) * cw + cc * 8 + row % 8] += v[q];
                        }
                    }
                }
            if (!direct) __syncthreads();
        }
        if (!direct)
            for (int q = threadIdx.x; q < na; q += CTHREADS) {
                const int c = c0 * 8 + q % cw, t = q / cw, tap = t % 9, o = o0 * 8 + t / 9;
                if (c < p.ci && o < p.co && tap % 3 >= kx0 && tap % 3 < kx0 + p.nkx)
                    atomicAdd(dw + ((long long)o * 9 + tap) * p.ci + c, acc[q]);
            }
    }
    if (!ok && err) atomicExch(err, NN_WAIT);
    tc_fence_before();
    __syncthreads();
    if (warp == EPW + 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(p.tcols) : "memory");
}

// ---------------------------------------------------------------------------
// Plans and launches
// ---------------------------------------------------------------------------
constexpr int SMS = 148;
int up_to(int v, int m) { return (v + m - 1) / m * m; }
int div_up(long long a, long long b) { return (int)((a + b - 1) / b); }
int tmem_cols(int n) { return n <= 32 ? 32 : n <= 64 ? 64 : n <= 128 ? 128 : n <= 256 ? 256 : 512; }

PFN_cuTensorMapEncodeTiled_v12000 encoder()
{
    static PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            p = nullptr;
        }
        return (PFN_cuTensorMapEncodeTiled_v12000)p;
    }();
    return fn;
}
bool encode(CUtensorMap* m, const void* base, int rank, const cuuint64_t* dims, const cuuint64_t* strides,
            const cuuint32_t* box)
{
    const cuuint32_t es[5] = {1, 1, 1, 1, 1};
    auto fn = encoder();
    return fn && fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void*>(base), dims, strides, box, es,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// chunk planes of an NHWC view (every `step`-th column and row from (dx, dy) on)
bool map_act(CUtensorMap* m, const Act& a, int step, int dx, int dy, int bw, int bh, int bch)
{
    const cuuint64_t px = (cuuint64_t)a.cs * 2;
    const cuuint64_t dims[5] = {8, (cuuint64_t)(a.w / step), (cuuint64_t)(a.h / step), (cuuint64_t)(a.c / 8), (cuuint64_t)a.nb};
    const cuuint64_t st[4] = {px * step, px * a.w * step, 16, px * a.w * a.h};
    const cuuint32_t box[5] = {8, (cuuint32_t)bw, (cuuint32_t)bh, (cuuint32_t)bch, 1};
    return encode(m, a.p + ((long long)dy * a.w + dx) * a.cs + a.off, 5, dims, st, box);
}
// rows of K-major weights [N][K] as chunk planes
bool map_w(CUtensorMap* m, const bf16* w, int N, int K, int bn)
{
    const cuuint64_t dims[3] = {8, (cuuint64_t)N, (cuuint64_t)(K / 8)};
    const cuuint64_t st[2] = {(cuuint64_t)K * 2, 16};
    const cuuint32_t box[3] = {8, (cuuint32_t)bn, 2};
    return encode(m, w, 3, dims, st, box);
}

// Tiles of a convolution over an nb x h x w output grid with N output channels and, per
// map, C input channels.  Columns: 128 at a time where the width is a multiple of 128
// (one MMA block per row); else whole rows (up to 254) one after the other in the MMA's
// 128 positions; else 126.  The number of rows ro, the output channels bn per CTA and
// whether the weights stay resident are chosen by a cost in cycles: staged 16-byte rows
// (about one a cycle), MMA time, epilogue, and waves of persistent CTAs.
//
// K order: tap by tap for 3x3 layers whose width is no multiple of 128 or with 8 input
// channels, channel group by group else, so that a layer's FP32 sums are taken in the
// same order for every tile shape; where a tile's groups do not fit in shared memory
// together (over about 256 channels), by group.
bool conv_plan(ConvP& best, size_t& smem, int& gx, int& gy, int nb, int h, int w, int N, int C, int nmap, bool three)
{
    ConvP p{};
    p.nb = nb;
    p.h = h;
    p.w = w;
    p.halo = three ? 1 : 0;
    p.nmap = nmap;
    p.C = C;
    p.G = (C + 15) / 16;
    p.pair8 = three && C == 8;
    p.taps = three ? (p.pair8 ? 5 : 9) : 1;
    p.nch = p.pair8 ? 1 : 2;
    const bool want_tap = three && (w % 128 != 0 || C % 16 != 0);
    const int GG = p.G * nmap, n16 = up_to(N, 16);
    const bool rowmode = w % 128 == 0;
    if (three) {
        p.txw = rowmode ? 128 : w <= 254 ? w : 126;
        p.wp = p.txw + 2;
    } else
        p.txw = p.wp = rowmode ? 128 : std::min(w, 256);
    p.tx = div_up(w, p.txw);
    double best_cost = 1e300;
    for (int ro = 1; ro <= 16; ro *= 2) {
        if (ro > 1 && ro / 2 >= h) break;
        p.ro = ro;
        p.rows = ro + 2 * p.halo + (p.pair8 ? 1 : 0);
        p.mstep = rowmode ? p.wp : 128;
        p.nblk = rowmode ? ro : div_up((long long)(ro - 1) * p.wp + p.txw, 128);
        p.ty = div_up(h, ro);
        if ((long long)p.tx * p.ty * nb > 0x7fffffff) continue;
        p.tiles = p.tx * p.ty * nb;
        p.plane = (uint32_t)(p.rows * p.wp * 16);
        p.aslot = up_to(p.nch * p.plane, 128);
        // the last block of positions may read past the last plane: keep that in bounds
        const int last = (p.nblk - 1) * p.mstep + 127 + (three ? 2 * p.wp + 2 : 0);
        const int over = std::max(0, last + 1 - p.rows * p.wp) * 16 + (p.pair8 ? p.wp * 16 : 0);
        for (int parts = 1; parts <= n16 / 16; parts++) {
            const int bn = up_to(div_up(n16, parts), 16);
            if (bn > 128 || p.nblk * bn > 512 || (parts > 1 && bn == up_to(div_up(n16, parts - 1), 16))) continue;
            p.bn = bn;
            p.wtap = 32u * bn;
            p.nbuf = 2 * p.nblk * bn <= 512 ? 2 : 1;
            p.tcols = tmem_cols(p.nbuf * p.nblk * bn);
            const int split = div_up(n16, bn);
            for (int stream = 0; stream < 2; stream++) {
                if (stream && p.pair8) continue;
                p.stream = stream;
                const size_t wres = stream ? 0 : (size_t)GG * p.taps * p.wtap;
                p.slot = p.aslot + (stream ? p.taps * p.wtap : 0);
                if (wres + over + 2 * (size_t)p.slot > SMEM_MAX) continue;
                int slots = (int)std::min<size_t>(MAXSLOT, (SMEM_MAX - wres - over) / p.slot);
                p.tapmajor = want_tap && GG <= slots;
                slots = std::min(slots, std::max(2, 3 * GG));
                p.slots = slots;
                const int per = std::max(1, SMS / split), waves = div_up(p.tiles, std::min(per, p.tiles));
                const double load = (double)GG * (p.nch * p.rows * p.wp + (stream ? p.taps * 2 * bn : 0));
                const double mma = (double)GG * p.taps * p.nblk * std::max(bn / 4.0, 12.0);
                const double epi = p.nblk * (bn / 8) * 60.0 / 2 + 200;
                const bool ahead = slots >= (p.tapmajor ? 2 * GG : 2);
                const double body = std::max(epi, ahead ? std::max(load, mma) : load + mma);
                const double tile = (p.nbuf == 2 ? body : std::max(load, mma + epi)) + 150;
                const double cost = waves * tile + load + mma + epi + 2500 + (double)wres / 32 +
                                    (want_tap && !p.tapmajor ? 1e9 : 0);
                if (cost < best_cost) {
                    best_cost = cost;
                    p.woff = (uint32_t)p.slots * p.slot;
                    best = p;
                    smem = (size_t)p.slots * p.slot + wres + over;
                    gx = std::min(per, p.tiles);
                    gy = split;
                }
            }
        }
    }
    return best_cost < 1e299;
}

template <class EP>
cudaError_t conv_launch(const Act* x, int nmap, int step, const bf16* w, int K, int nb, int h, int wd, int N, bool three,
                        const EP& ep, int* err, cudaStream_t st)
{
    ConvP p;
    size_t smem;
    int gx, gy;
    if (!conv_plan(p, smem, gx, gy, nb, h, wd, N, x->c, nmap, three)) return cudaErrorInvalidValue;
    ConvMaps maps;
    for (int q = 0; q < nmap; q++)
        if (!map_act(&maps.x[q], *x, step, q & 1, q >> 1, p.wp, p.rows, p.nch)) return cudaErrorInvalidValue;
    for (int q = nmap; q < 4; q++) maps.x[q] = maps.x[0];
    if (!map_w(&maps.w, w, N, K, p.bn)) return cudaErrorInvalidValue;
    static unsigned long long opted = 0;
    const cudaError_t e = ertm::smem_opt_in(k_conv<EP>, SMEM_MAX, &opted);
    if (e != cudaSuccess) return e;
    return ertm::launch_pdl(k_conv<EP>, dim3(gx, gy), dim3(CTHREADS), smem, st, maps, p, ep, err);
}

// Tiles of a weight gradient.  3x3: rr rows of dy against rr + 2 of x; more rows re-read
// less of x and waste fewer row pairs but need TMEM (mb * n columns per kx, 512 in all)
// and shared memory for two stages or more.
bool wgrad_plan(WgP& best, size_t& smem, dim3& grid, int nb, int h, int w, int ci, int co, bool up)
{
    WgP p{};
    p.nb = nb;
    p.h = h;
    p.w = w;
    p.ci = ci;
    p.co = co;
    p.up = up;
    const int c8 = ci / 8, o8 = co / 8;
    double best_cost = 1e300;
    for (int tw = 128; tw >= 16; tw /= 2) {
        if (tw > 16 && tw / 2 >= up_to(w, 16)) continue;
        p.tw = tw;
        p.tx = div_up(w, tw);
        for (int rr = 1; rr <= 12; rr++) {
            if (rr > h && rr > 1) break;
            p.rr = rr;
            p.ty = div_up(h, rr);
            p.units = p.tx * p.ty * nb;
            for (int nkx = up ? 1 : 3; nkx >= 1; nkx -= 2) {
                p.nkx = nkx;
                p.kgroups = up ? 1 : 3 / nkx;
                for (int cdiv = 1; cdiv <= c8; cdiv *= 2)
                    for (int odiv = 1; odiv <= o8; odiv *= 2) {
                        p.CC = div_up(c8, cdiv);
                        p.OC = div_up(o8, odiv);
                        if (up) {
                            p.CC = up_to(p.CC, 2);          // N in multiples of 16
                            p.jr = rr;
                            p.planes = 4 * p.OC;
                            p.n = 8 * p.CC;
                            p.pitchA = p.pitchB = (uint32_t)(rr * tw * 16);
                            p.ksteps = rr * tw / 16;
                            p.abytes = (uint32_t)p.planes * p.pitchA;
                            p.bbytes = (uint32_t)p.CC * p.pitchB;
                        } else {
                            if ((p.OC * rr) % 2) p.OC++;
                            p.jr = rr + 2;
                            p.planes = p.CC * p.jr;
                            p.n = 8 * p.OC * rr;
                            p.pitchA = (uint32_t)((tw + 2) * 16);
                            p.pitchB = (uint32_t)(tw * 16);
                            p.ksteps = tw / 16;
                            p.abytes = up_to(p.planes * p.pitchA, 128);
                            p.bbytes = (uint32_t)(p.OC * rr) * p.pitchB;
                        }
                        p.mb = div_up(p.planes, 16);
                        const int cols = p.mb * p.nkx * p.n;
                        if (p.n > 256 || cols > 512 || p.CC > 256 || p.OC > 256) continue;
                        p.stage = up_to(p.abytes + p.bbytes, 128);
                        // MMA blocks are 16 planes: the last may read past the staged ones
                        const int over = std::max(0, (int)(p.mb * 16 - p.planes) * (int)p.pitchA + 64 - (int)p.bbytes);
                        if (2 * (size_t)p.stage + over > SMEM_MAX) continue;
                        const int stages = std::min(8, (int)((SMEM_MAX - over) / p.stage));
                        const size_t accb = up || rr == 1 ? 0 : (size_t)p.OC * 8 * 9 * p.CC * 8 * 4;
                        if (accb > SMEM_MAX) continue;
                        p.stages = stages;
                        p.tcols = tmem_cols(cols);
                        p.cb = div_up(c8, p.CC);
                        const int others = p.kgroups * p.cb * div_up(o8, p.OC);
                        const int px = up ? rr * tw : tw;        // accumulator chain per unit
                        const int least = div_up((long long)p.units * px, 4096);
                        const int splits = std::min(p.units, std::max(std::max(1, SMS / others), least));
                        const int waves = div_up((long long)splits * others, SMS);
                        const double load = up ? (double)(p.planes + p.CC) * rr * tw
                                               : (double)p.planes * (tw + 2) + (double)p.OC * rr * tw;
                        const double mma = (double)p.ksteps * p.nkx * p.mb * std::max(p.n / 4.0, 16.0);
                        const double sums = up ? (double)p.mb * 16 * p.n : 9.0 * p.CC * 8 * p.OC * 8 * p.nkx / 3;
                        const double epi = 3000 + sums / 24 * (up || rr == 1 ? 2 : 1) + (double)cols * (rr > 1 && !up ? 4 : 2);
                        const double cost = waves * (div_up(p.units, splits) * (std::max(load, mma) + 250) + load + epi);
                        if (cost < best_cost) {
                            best_cost = cost;
                            best = p;
                            smem = std::max((size_t)stages * p.stage + over, accb);
                            grid = dim3(splits, p.kgroups, p.cb * div_up(o8, p.OC));
                        }
                    }
            }
        }
    }
    return best_cost < 1e299;
}

cudaError_t wgrad_launch(const Act& x, const Act& dy, float* dw, bool up, int* err, cudaStream_t st)
{
    WgP p;
    size_t smem;
    dim3 grid;
    if (!wgrad_plan(p, smem, grid, x.nb, x.h, x.w, x.c, dy.c, up)) return cudaErrorInvalidValue;
    WgMaps maps;
    bool ok = true;
    if (up) {
        for (int q = 0; q < 4; q++) ok = ok && map_act(&maps.a[q], dy, 2, q & 1, q >> 1, p.tw, p.rr, p.OC);
        ok = ok && map_act(&maps.b, x, 1, 0, 0, p.tw, p.rr, p.CC);
    } else {
        ok = map_act(&maps.a[0], x, 1, 0, 0, p.tw + 2, p.jr, p.CC);
        for (int q = 1; q < 4; q++) maps.a[q] = maps.a[0];
        ok = ok && map_act(&maps.b, dy, 1, 0, 0, p.tw, p.rr, p.OC);
    }
    if (!ok) return cudaErrorInvalidValue;
    static unsigned long long opted = 0;
    const cudaError_t e = ertm::smem_opt_in(k_wgrad, SMEM_MAX, &opted);
    if (e != cudaSuccess) return e;
    return ertm::launch_pdl(k_wgrad, grid, dim3(CTHREADS), smem, st, maps, p, dw, err);
}

}  // namespace

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
extern "C" {

int ertm_nn_conv3x3(const ertm_nn_act* x, const void* w, const float* bias, const ertm_nn_act* y, int relu,
                    float* y32, int* err, void* stream)
{
    if (!act_ok(x) || !aligned16(w) || !y || (!y32 && !act_ok(y))) return ERTM_EINVAL;
    if (y->n != x->n || y->h != x->h || y->w != x->w) return ERTM_EINVAL;
    const Act xa = act_of(x);
    const int N = y->c, K = 9 * x->c;
    const bf16* wb = reinterpret_cast<const bf16*>(w);
    cudaStream_t st = (cudaStream_t)stream;
    if (y32) {
        EpiF32 ep{y32, y->cstride, N, y->cstride % 4 == 0 && aligned16(y32), bias};
        return rc_of(conv_launch(&xa, 1, 1, wb, K, x->n, x->h, x->w, N, true, ep, err, st));
    }
    EpiAct ep{reinterpret_cast<bf16*>(const_cast<void*>(y->data)), y->cstride, y->coff, N, relu, bias};
    return rc_of(conv_launch(&xa, 1, 1, wb, K, x->n, x->h, x->w, N, true, ep, err, st));
}

int ertm_nn_conv3x3_dgrad(const ertm_nn_act* dy, const void* wflip, const ertm_nn_act* dx, const ertm_nn_act* mask,
                          int* err, void* stream)
{
    if (!act_ok(dy) || !aligned16(wflip) || !act_ok(dx) || !same_grid(dy, dx)) return ERTM_EINVAL;
    if (!mask_ok(mask, dx)) return ERTM_EINVAL;
    const Act da = act_of(dy);
    EpiGrad ep{reinterpret_cast<bf16*>(const_cast<void*>(dx->data)), dx->cstride, dx->coff, dx->c,
               mask ? reinterpret_cast<const bf16*>(mask->data) : nullptr};
    return rc_of(conv_launch(&da, 1, 1, reinterpret_cast<const bf16*>(wflip), 9 * dy->c, dy->n, dy->h, dy->w, dx->c, true,
                             ep, err, (cudaStream_t)stream));
}

int ertm_nn_conv3x3_wgrad(const ertm_nn_act* x, const ertm_nn_act* dy, float* dw, int splitk, int* err, void* stream)
{
    (void)splitk;   // a hint: the plan splits the pixels by itself
    if (!act_ok(x) || !act_ok(dy) || !dw) return ERTM_EINVAL;
    Act da = act_of(dy);            // dy's pixels are taken in x's grid, in order
    da.nb = x->n;
    da.h = x->h;
    da.w = x->w;
    return rc_of(wgrad_launch(act_of(x), da, dw, false, err, (cudaStream_t)stream));
}

int ertm_nn_up2(const ertm_nn_act* x, const void* u, const float* bias, const ertm_nn_act* y, int relu, int* err,
                void* stream)
{
    if (!act_ok(x) || !aligned16(u) || !act_ok(y) || y->h != 2 * x->h || y->w != 2 * x->w || y->n != x->n)
        return ERTM_EINVAL;
    if (x->coff != 0 || x->cstride != x->c) return ERTM_EINVAL;
    const Act xa = act_of(x);
    EpiUp2 ep{reinterpret_cast<bf16*>(const_cast<void*>(y->data)), y->cstride, y->coff, y->c, x->h, x->w, relu, bias};
    return rc_of(conv_launch(&xa, 1, 1, reinterpret_cast<const bf16*>(u), x->c, x->n, x->h, x->w, 4 * y->c, false, ep, err,
                             (cudaStream_t)stream));
}

int ertm_nn_up2_dgrad(const ertm_nn_act* dy, const void* ut, const ertm_nn_act* dx, const ertm_nn_act* mask,
                      int* err, void* stream)
{
    if (!act_ok(dy) || !aligned16(ut) || !act_ok(dx) || dy->h != 2 * dx->h || dy->w != 2 * dx->w || dy->n != dx->n ||
        !mask_ok(mask, dx))
        return ERTM_EINVAL;
    const Act da = act_of(dy);
    EpiGrad ep{reinterpret_cast<bf16*>(const_cast<void*>(dx->data)), dx->cstride, dx->coff, dx->c,
               mask ? reinterpret_cast<const bf16*>(mask->data) : nullptr};
    return rc_of(conv_launch(&da, 4, 2, reinterpret_cast<const bf16*>(ut), 4 * dy->c, dx->n, dx->h, dx->w, dx->c, false, ep,
                             err, (cudaStream_t)stream));
}

int ertm_nn_up2_wgrad(const ertm_nn_act* x, const ertm_nn_act* dy, float* du, int splitk, int* err, void* stream)
{
    (void)splitk;
    if (!act_ok(x) || !act_ok(dy) || !du || dy->h != 2 * x->h || dy->w != 2 * x->w) return ERTM_EINVAL;
    Act da = act_of(dy);
    da.nb = x->n;
    return rc_of(wgrad_launch(act_of(x), da, du, true, err, (cudaStream_t)stream));
}

}  // extern "C"
