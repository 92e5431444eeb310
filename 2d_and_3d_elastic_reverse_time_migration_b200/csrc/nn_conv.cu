// The U-Net's convolutions on the tensor cores: 3x3 and 2x2 transposed convolutions,
// their input gradients and their weight gradients (BF16 operands, FP32 accumulation in
// tensor memory).
//
// Operands are staged by TMA in blocks of cb = 16, 32 or 64 channels: one 4D box (cb
// channels, columns, rows, image) of the NHWC view, zero outside the image, lands in shared
// memory as [row][column][2 cb bytes] with the 32-, 64- or 128-byte swizzle.  The swizzle
// is a function of the shared-memory address alone, for TMA as for the tensor core, so
// the staged block is read in place and from any pixel on.  (Channel counts that are no
// multiple of 16 are staged as planes of 16-byte chunks without swizzle, boxes of 8
// channels, [chunk][row][column][16 B]: more lines for TMA to move.)
//   * as a K-major operand (rows = pixels, K = channels): 128 consecutive staged pixels
//     are the M side, and a tap (ky, kx) of the 3x3 stencil is the same planes read
//     ky rows and kx pixels further.  An image row is staged with its padding column on
//     either side, so rows follow one another with a pitch of Wp pixels and 128
//     consecutive positions may run over several rows of a narrow image (the two
//     padding positions per row are computed and not stored);
//   * as an MN-major operand (rows = channels, K = pixels): the weight gradient's two
//     sides.  The (block, row) pairs are the M side of x and the N side of dy; one MMA
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
// 14.08 -> 2.32 ms, one 256 x 512 image forward 595 -> 157 us (bit-identical), a single
// 32 -> 48 layer on 5 x 61 x 107 with its gradients 264 -> 50 us.  Of the batch's way:
// 16-byte planes and one thread computing every descriptor 3.86 ms; swizzled blocks 4.07
// (no line bound yet, more arithmetic per MMA), the warp computing them in uniform registers
// 3.60, MMA tables 2.86, four epilogue warps per lane quarter with the mask read ahead and
// the 2x2 sums through shared memory 2.53, the bias gradients taken by the weight gradients'
// idle warps and one call per pass 2.32 (the 18 separate bias kernels took 212 us).
//
// What bounds them: at 16-32 channels a layer moves 64-200 bytes per pixel for 5-18 kFLOP,
// the HBM side; next to it the lines of the boxes (TMA moves one in 1.6, 2.7, 3.4 or 7
// cycles for 16, 32, 64 or 128 bytes) and the MMAs (40 cycles at least, whatever N).
#include <algorithm>

#include "nn_common.cuh"

#include <cudaTypedefs.h>

namespace {

// ---------------------------------------------------------------------------
// Epilogues: at(m) is where output row m goes (once per lane and block), then 8
// consecutive columns n0..n0+7 at a time (n0 % 8 == 0); pre() loads what the epilogue
// needs besides the accumulators, ahead of them
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
    typedef long long At;
    __device__ __forceinline__ At at(int m) const { return (long long)m * cs + off; }
    __device__ __forceinline__ Pre pre(At, int) const { return Pre(); }
    __device__ __forceinline__ void operator()(At a, int n0, const float* v, const Pre&) const
    {
        if (n0 >= N) return;
        float t[8];
#pragma unroll
        for (int q = 0; q < 8; q++) {
            t[q] = v[q] + (bias ? __ldg(bias + n0 + q) : 0.f);
            if (relu) t[q] = fmaxf(t[q], 0.f);
        }
        *reinterpret_cast<uint4*>(y + a + n0) = pack8(t);
    }
};

// FP32 NHWC output without activation (network output)
struct EpiF32 {
    float* y;
    int cs, N, vec;          // vec: 16-byte stores are aligned
    const float* bias;
    typedef NoPre Pre;
    typedef long long At;
    __device__ __forceinline__ At at(int m) const { return (long long)m * cs; }
    __device__ __forceinline__ Pre pre(At, int) const { return Pre(); }
    __device__ __forceinline__ void operator()(At a, int n0, const float* v, const Pre&) const
    {
        float* d = y + a + n0;
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
    typedef long long At;
    __device__ __forceinline__ At at(int m) const { return (long long)m * cs + off; }
    __device__ __forceinline__ Pre pre(At a, int n0) const
    {
        if (!mask || n0 >= N) return make_uint4(0, 0, 0, 0);
        return __ldg(reinterpret_cast<const uint4*>(mask + a + n0));
    }
    __device__ __forceinline__ void operator()(At a, int n0, const float* v, const Pre& k) const
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
        *reinterpret_cast<uint4*>(dx + a + n0) = pack8(t);
    }
};

// transposed 2x2 stride-2 convolution: column n = (a*2 + b) * C + o scatters to
// the high-resolution pixel (2i+a, 2j+b) of low-resolution row m; C % 8 == 0
struct EpiUp2 {
    bf16* y;
    int cs, off, C, lh, lw, relu;
    const float* bias;
    typedef NoPre Pre;
    typedef long long At;
    __device__ __forceinline__ At at(int m) const
    {
        const int j = m % lw, q2 = m / lw, i = q2 % lh, nb = q2 / lh;
        return ((long long)(nb * 2 * lh + 2 * i) * 2 * lw + 2 * j) * cs + off;
    }
    __device__ __forceinline__ Pre pre(At, int) const { return Pre(); }
    __device__ __forceinline__ void operator()(At a, int n0, const float* v, const Pre&) const
    {
        if (n0 >= 4 * C) return;
        const int ab = n0 / C, o = n0 - ab * C;
        float t[8];
#pragma unroll
        for (int q = 0; q < 8; q++) {
            t[q] = v[q] + (bias ? __ldg(bias + o + q) : 0.f);
            if (relu) t[q] = fmaxf(t[q], 0.f);
        }
        *reinterpret_cast<uint4*>(y + a + (long long)((ab >> 1) * 2 * lw + (ab & 1)) * cs + o) = pack8(t);
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
__device__ __forceinline__ void tma4(void* dst, const CUtensorMap* m, int c, int x, int y, int n, uint64_t* bar)
{
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4, %5}], [%6];\n" ::"r"(su32(dst)),
        "l"(m), "r"(c), "r"(x), "r"(y), "r"(n), "r"(su32(bar))
        : "memory");
}
__device__ __forceinline__ void tma2(void* dst, const CUtensorMap* m, int k, int r, uint64_t* bar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3}], [%4];\n" ::"r"(su32(dst)),
        "l"(m), "r"(k), "r"(r), "r"(su32(bar))
        : "memory");
}
// descriptor layout code of blocks of cb channels (0: 16-byte chunks, no swizzle)
__host__ __device__ constexpr uint64_t swizzle_code(int cb)
{
    return cb == 64 ? 2ull << 61 : cb == 32 ? 4ull << 61 : cb == 16 ? 6ull << 61 : 0ull;
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

__device__ __forceinline__ bool all_lanes(bool v) { return __all_sync(0xffffffffu, v); }
// true in one lane of a converged warp
__device__ __forceinline__ bool elect1()
{
    uint32_t v;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(v));
    return v != 0;
}

// One MMA of a tile: a = offset of its A operand in the slot (low half) and what it adds to
// the descriptor's LBO (high half), w = offset of its B operand (low) and accumulator
// column (high); offsets in units of 16 bytes.  Everything that an MMA's descriptors need
// an index computation for is in the table: the one thread that issues has a few
// instructions between two MMAs (40-65 cycles each, what the tensor core takes for M = 128
// and N = 16 .. 128; with the index arithmetic in its loop it was 95-280).
struct MmaEntry {
    uint32_t a, w;
};
// n entries from e; the first `fresh` of them start their accumulators
__device__ __forceinline__ void issue(const MmaEntry* e, int n, uint32_t td, uint64_t dA, uint64_t dB, uint32_t idesc,
                                      int fresh)
{
    auto one = [&](const MmaEntry& m, uint32_t acc) {
        umma(td + (m.w >> 16), dA + m.a, dB + (m.w & 0xffffu), idesc, acc);
    };
    int i = 0;
    for (; i < fresh; i++) one(e[i], 0u);
    for (; i + 4 <= n; i += 4) {
        MmaEntry m[4];
#pragma unroll
        for (int q = 0; q < 4; q++) m[q] = e[i + q];
#pragma unroll
        for (int q = 0; q < 4; q++) one(m[q], 1u);
    }
    for (; i < n; i++) one(e[i], 1u);
}

constexpr int EPW = 16;                // epilogue warps: four per quarter of the TMEM lanes
constexpr int CTHREADS = 32 * (EPW + 2);
constexpr int MAXSLOT = 16;
constexpr int SMEM_MAX = 220 * 1024;   // dynamic shared memory a CTA may take
constexpr int ZEROS = 128 * 16;        // one 16-byte chunk of each of an MMA's 128 rows

// Tile plan of a convolution launch
struct ConvP {
    int nb, h, w;                 // output grid
    int wp, txw, ro, rows;        // staged pitch; output columns and rows of a tile; staged rows
    int halo, tx, ty, tiles;      // 1: staged rows and columns around the tile; tiles per row, row groups, tiles
    int nblk, mstep;              // 128-row MMA blocks per tile; positions from one to the next
    int C, nmap, taps;            // channels per map, maps, taps
    int cb, B;                    // channels per staged block (0: chunk planes of 16 or 8 channels), blocks per map
    int nch;                      // chunk planes per block
    int tapmajor, pair8, stream;  // K order; 8-channel taps in pairs; weights staged with each block
    int slots, nbuf, bn, tcols;
    uint32_t pitch;               // bytes of a staged pixel
    uint32_t plane, abytes, aslot, slot;   // bytes: a chunk plane, a box, a slot's input part, a slot
    uint32_t zeros;               // pair8: offset of a slot's ZEROS bytes of zeros
    uint32_t wtap;                // chunk planes: bytes of the weights of one block and tap
    uint32_t woff, wbytes;        // resident weights: shared-memory offset, bytes
    int groups, entries;          // 16-channel groups and MMAs of a tile (streamed: of a block)
    uint32_t toff;                // shared-memory offset of the MMA table
};
struct ConvMaps {
    CUtensorMap x[4];             // the input (2x2 input gradient: one per output phase)
    CUtensorMap w;                // weights [N][K]: 64 K x bn rows (chunk planes: 8 K x bn rows x 2 chunks)
};

// Warps 0-15: epilogue, 16: TMA, 17: MMA.  K runs over groups of 16 channels and, inside a
// group, over its taps; with `tapmajor` over the taps and inside a tap over the groups
// (all blocks of a tile staged at once): the two orders in which FP32 sums of these
// layers have always been taken, by width and channel count (see conv_plan).
template <class EP>
__global__ void __launch_bounds__(CTHREADS, 1) k_conv(const __grid_constant__ ConvMaps maps,
                                                      const __grid_constant__ ConvP p, const EP ep, int* err)
{
    extern __shared__ __align__(1024) uint8_t sm[];
    __shared__ uint64_t full[MAXSLOT], empty[MAXSLOT], tfull[2], tempty[2], wfull, done;
    __shared__ uint32_t tmem_s;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int n0 = blockIdx.y * p.bn;
    const int BB = p.nmap * p.B;
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
    if (p.pair8) {
        for (int q = threadIdx.x; q < p.slots * (ZEROS / 16); q += CTHREADS)
            *reinterpret_cast<uint4*>(sm + (size_t)(q / (ZEROS / 16)) * p.slot + p.zeros + q % (ZEROS / 16) * 16) =
                make_uint4(0, 0, 0, 0);
        proxy_fence();
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
                expect_tx(&wfull, p.wbytes);
                if (p.cb) {
                    for (uint32_t o = 0, k = 0; o < p.wbytes; o += 128u * p.bn, k += 64)
                        tma2(sm + p.woff + o, &maps.w, k, n0, &wfull);
                } else {
                    for (int bb = 0; bb < BB; bb++)
                        for (int t = 0; t < p.taps; t++) {
                            const int m = bb / p.B, g = bb - m * p.B;
                            const int kc = p.pair8 ? 2 * t : ((m + t) * p.C >> 3) + 2 * g;
                            tma3w(sm + p.woff + (uint32_t)(bb * p.taps + t) * p.wtap, &maps.w, 0, n0, kc, &wfull);
                        }
                }
                wis = true;
            }
            for (int u = blockIdx.x; u < p.tiles && ok; u += gridDim.x) {
                const int xt = u % p.tx, q = u / p.tx, yt = q % p.ty, nb = q / p.ty;
                const int x0 = xt * p.txw - p.halo, y0 = yt * p.ro - p.halo;
                for (int bb = 0; bb < BB; bb++) {
                    const int sl = issued % p.slots, use = issued / p.slots;
                    if (use > 0 && !mbar_wait(&empty[sl], (use - 1) & 1)) {
                        ok = false;
                        break;
                    }
                    uint8_t* d = sm + (size_t)sl * p.slot;
                    const int m = bb / p.B, g = bb - m * p.B;
                    expect_tx(&full[sl], p.abytes + (p.stream ? p.taps * p.wtap : 0u));
                    if (p.cb) tma4(d, &maps.x[m], g * p.cb, x0, y0, nb, &full[sl]);
                    else tma5(d, &maps.x[m], 0, x0, y0, 2 * g, nb, &full[sl]);
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
        // The tile's MMAs as a table, built once by the warp (see MmaEntry); one elected lane
        // issues them from it.  K order: by 16-channel group, or by tap (tapmajor).
        const bool el = elect1();
        const uint32_t idesc = idesc_bf16(p.bn);
        const uint32_t p16 = p.pitch >> 4, sm16 = su32(sm) >> 4, slot16 = p.slot >> 4;
        MmaEntry* tab = reinterpret_cast<MmaEntry*>(sm + p.toff);
        for (int i = lane; i < p.entries; i += 32) {
            const int b = i % p.nblk, e = i / p.nblk;
            // group gg of the tile's (of the block's, streamed), tap t
            const int t = p.tapmajor ? e / p.groups : e % p.taps, gg = p.tapmajor ? e - t * p.groups : e / p.taps;
            uint32_t a = 0, w = 0, lbo = 0;
            if (p.cb) {
                const int gm = p.C / 16, m = gg / gm, c = 16 * (gg - m * gm), k = (m + t) * p.C + c;
                a = (c % p.cb) / 8;
                w = (k >> 6) * (8 * p.bn) + ((k & 63) >> 3);
            } else
                w = (p.stream ? (p.aslot >> 4) : 0) + (gg * p.taps + t) * (p.wtap >> 4);
            if (p.pair8) {
                // K = taps 2t, 2t+1 of the one chunk.  The ninth has zero weights beside it, and
                // zeros for pixels: a pixel there could be infinite, and its product NaN.
                const int ta = 2 * t, tb = ta + 1;
                a = (ta / 3) * p.wp + ta % 3;
                lbo = tb < 9 ? (tb / 3) * p.wp + tb % 3 - a : (p.zeros >> 4) - (a + b * p.mstep);
            } else if (p.halo)
                a += ((t / 3) * p.wp + t % 3) * p16;
            tab[i] = MmaEntry{a + b * p.mstep * p16 | lbo << 16, w | (uint32_t)(b * p.bn) << 16};
        }
        __syncwarp();
        const uint64_t dA = sdesc(0, p.cb ? 16 : p.pair8 ? 0 : p.plane, p.cb ? 8 * p.pitch : 128) | swizzle_code(p.cb);
        const uint64_t dB = p.cb ? sdesc(su32(sm) + p.woff, 16, 1024) | swizzle_code(64)
                                 : sdesc(p.stream ? 0 : su32(sm) + p.woff, p.bn * 16);
        const int per = p.entries / (p.stream ? 1 : BB);     // entries of a block (swizzled blocks: all but the last)
        int used = 0, nt = 0;
        if (!p.stream) ok = all_lanes(mbar_wait(&wfull, 0));
        for (int u = blockIdx.x; u < p.tiles && ok; u += gridDim.x, nt++) {
            const int buf = nt % p.nbuf, use = nt / p.nbuf;
            if (use > 0 && !all_lanes(mbar_wait(&tempty[buf], (use - 1) & 1))) {
                ok = false;
                break;
            }
            tc_fence_after();
            const uint32_t td = tmem + (uint32_t)(buf * p.nblk * p.bn);
            if (p.tapmajor) {
                // every block of the tile, then tap by tap over them: the table names the group
                for (int g = 0; g < BB && ok; g++)
                    ok = all_lanes(mbar_wait(&full[(used + g) % p.slots], ((used + g) / p.slots) & 1));
                if (!ok) break;
                tc_fence_after();
                const int s0 = used % p.slots, bg = p.cb ? p.cb / 16 : 1, n = p.nblk;
                if (el) {
                    // runs of groups in one block: bg (the last block of a map may have fewer)
                    int i = 0;
                    for (int t = 0; t < p.taps; t++)
                        for (int g = 0, sl = s0, left = p.groups; g < BB; g++, sl = sl + 1 == p.slots ? 0 : sl + 1) {
                            const int m = min(bg, left) * n;
                            left -= bg;
                            issue(tab + i, m, td, dA + sm16 + sl * slot16,
                                  p.stream ? dB + sm16 + sl * slot16 : dB, idesc, i == 0 ? n : 0);
                            i += m;
                        }
                    for (int g = 0, sl = s0; g < BB; g++, sl = sl + 1 == p.slots ? 0 : sl + 1) umma_commit(&empty[sl]);
                }
                used += BB;
            } else {
                int i = 0;
                const int gm = p.C / 16, bg = p.cb / 16;
                for (int g = 0, left = gm; g < BB; g++, used++) {
                    const int sl = used % p.slots;
                    if (!all_lanes(mbar_wait(&full[sl], (used / p.slots) & 1))) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    // swizzled blocks: up to bg groups, the last of a map may have fewer
                    const int m = p.cb ? min(bg, left) * p.taps * p.nblk : per;
                    left = left <= bg ? gm : left - bg;
                    if (el) {
                        const uint32_t a16 = sm16 + sl * slot16;
                        issue(tab + (p.stream ? 0 : i), m, td, dA + a16, p.stream ? dB + a16 : dB, idesc, g == 0 ? p.nblk : 0);
                        umma_commit(&empty[sl]);
                    }
                    i += m;
                }
                if (!ok) break;
            }
            if (el) umma_commit(&tfull[buf]);
        }
        if (el) umma_commit(&done);       // every MMA issued has completed before TMEM is freed
        if (!mbar_wait(&done, 0)) ok = false;
        __syncwarp();
    } else {
        const int quad = warp & 3, set = warp >> 2;
        // this lane's output row of block b of tile u (place), or none
        struct Place {
            typename EP::At at;
            bool in;
        };
        auto place = [&](int u, int b) {
            const int xt = u % p.tx, q = u / p.tx, yt = q % p.ty, nb = q / p.ty;
            const int pos = b * p.mstep + quad * 32 + lane;
            const int r = pos / p.wp, xx = pos - r * p.wp;
            const int gx = xt * p.txw + xx, gy = yt * p.ro + r;
            Place l;
            l.in = u < p.tiles && b < p.nblk && xx < p.txw && gx < p.w && r < p.ro && gy < p.h &&
                   (p.mstep == 128 || r == b);
            l.at = ep.at(l.in ? (nb * p.h + gy) * p.w + gx : 0);
            return l;
        };
        auto load = [&](const Place& l, int c, typename EP::Pre* pre) {
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (l.in && c + 8 * k < p.bn) pre[k] = ep.pre(l.at, n0 + c + 8 * k);
        };
        constexpr int SETS = EPW / 4;
        int nt = 0;
        // the first 32 columns' pre-loads run one block ahead
        Place cur = place(blockIdx.x, set);
        typename EP::Pre nxt[4];
        load(cur, 0, nxt);
        for (int u = blockIdx.x; u < p.tiles && ok; u += gridDim.x, nt++) {
            const int buf = nt % p.nbuf, use = nt / p.nbuf;
            ok = all_lanes(mbar_wait(&tfull[buf], use & 1));
            if (!ok) break;
            tc_fence_after();
            for (int b = set; b < p.nblk; b += SETS) {
                const Place l = cur;
                typename EP::Pre pre[4];
#pragma unroll
                for (int k = 0; k < 4; k++) pre[k] = nxt[k];
                cur = b + SETS < p.nblk ? place(u, b + SETS) : place(u + gridDim.x, set);
                load(cur, 0, nxt);
                const uint32_t td = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)((buf * p.nblk + b) * p.bn);
                for (int c = 0; c < p.bn; c += 32) {
                    if (c) load(l, c, pre);
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
                            if (l.in) ep(l.at, n0 + c + 8 * k, f, pre[k]);
                        }
                }
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
    int ci, co;
    int cx, cy;                   // channels per staged block of x and of dy (8: chunk planes)
    int CB, OB;                   // blocks of x and dy that a CTA stages
    int cparts;                   // such sets of x (grid z = cparts x sets of dy)
    int atoms;                    // M side: staged (block, row) pairs
    int mb, n, nkx, kgroups;      // MMA blocks, N, kx windows per CTA, groups of them
    int ksteps;
    uint32_t pitchA, pitchB;      // bytes from one (block, row) pair to the next
    uint32_t atx, abytes, bbytes, stage;
    uint32_t toff;                // shared-memory offset of the MMA table
    int stages, tcols;
    int up;                       // 2x2 transposed convolution: M = (phase, dy block), N = x block
    int staged;                   // its sums pass through shared memory
};
struct WgMaps {
    CUtensorMap a[4], b;
};
struct WgSrc {
    Act x, dy;
};

// A 3x3 weight's sum over the CTA's tiles, product by product
__device__ float wgrad_sum(const WgP& p, const WgSrc& a, int c, int o, int tap)
{
    const int ky = tap / 3, kx = tap - 3 * ky;
    float s = 0.f;
    for (int u = blockIdx.x; u < p.units; u += gridDim.x) {
        const int xt = u % p.tx, q = u / p.tx, yt = q % p.ty, nb = q / p.ty;
        const int bottom = min(p.h, (yt + 1) * p.rr), end = min(p.w, (xt + 1) * p.tw);
        for (int y = yt * p.rr; y < bottom; y++) {
            const int xy = y + ky - 1;
            for (int i = xt * p.tw; i < end; i++) {
                const int xc = i + kx - 1;
                const float d = __bfloat162float(a.dy.p[((long long)(nb * p.h + y) * p.w + i) * a.dy.cs + a.dy.off + o]);
                float v = 0.f;
                if (xy >= 0 && xy < p.h && xc >= 0 && xc < p.w)
                    v = __bfloat162float(a.x.p[((long long)(nb * p.h + xy) * p.w + xc) * a.x.cs + a.x.off + c]);
                s += v * d;
            }
        }
    }
    return s;
}
// The weights whose accumulator is NaN, once more and without the tensor core.  dy is staged
// as zeros past the last column and row, where the first tap of a row or column still meets
// x's last one: an infinite activation there makes a product NaN that the gradient does
// not have.  Out of line, and after the sums that are none: calls among them took registers
// from every launch (loss and gradients of a 16 x 256 x 512 batch 2.31 -> 2.40 ms).
__device__ __noinline__ void wgrad_repair(const WgP& p, const WgSrc& src, const float* acc, uint32_t tmem, float* dw)
{
    const int kx0 = blockIdx.y * p.nkx;
    const int c0 = (int)(blockIdx.z % p.cparts) * p.CB * p.cx, o0 = (int)(blockIdx.z / p.cparts) * p.OB * p.cy;
    auto add = [&](int c, int o, int tap) {
        atomicAdd(dw + ((long long)o * 9 + tap) * p.ci + c, wgrad_sum(p, src, c, o, tap));
    };
    if (p.rr > 1) {                      // sums in shared memory, as k_wgrad leaves them
        const int cw = p.CB * p.cx, na = p.OB * p.cy * 9 * cw;
        for (int q = threadIdx.x; q < na; q += CTHREADS) {
            const int c = c0 + q % cw, t = q / cw, tap = t % 9, o = o0 + t / 9;
            if (c < p.ci && o < p.co && tap % 3 >= kx0 && tap % 3 < kx0 + p.nkx && acc[q] != acc[q]) add(c, o, tap);
        }
        return;
    }
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), quad = warp & 3;
    if (warp >= EPW) return;
    for (int t = warp >> 2; t < p.nkx * p.mb; t += EPW / 4) {
        const int k = t / p.mb, b = t - k * p.mb, row = quad * 32 + (threadIdx.x & 31);
        const int at = b * (128 / p.cx) + row / p.cx, cbk = at / p.jr, ky = at - cbk * p.jr;
        const int c = c0 + cbk * p.cx + row % p.cx, tap = ky * 3 + kx0 + k;
        const bool in = at < p.atoms && ky < 3 && kx0 + k < 3 && c < p.ci;
        for (int n8 = 0; n8 < p.n; n8 += 8) {
            float v[8];
            __syncwarp();
            tmem_ld8(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(t * p.n + n8), v);
#pragma unroll
            for (int q = 0; q < 8; q++)
                if (in && o0 + n8 + q < p.co && v[q] != v[q]) add(c, o0 + n8 + q, tap);
        }
    }
}

// Partial sums of a CTA's tiles stay in TMEM (3x3: one accumulator per kx, lanes (x
// chunk, x row j, channel), columns (dy chunk, dy row r, channel)); at the end the lanes
// and columns with j - r = ky in 0..2 are the gradient of tap ky, summed over r in shared
// memory and added to dw once per CTA.  A CTA takes at most 4096 pixels per accumulator
// chain, unless the caller bounds the splits.
__global__ void __launch_bounds__(CTHREADS, 1) k_wgrad(const __grid_constant__ WgMaps maps,
                                                       const __grid_constant__ WgP p,
                                                       const __grid_constant__ WgSrc src, float* __restrict__ dw,
                                                       float* __restrict__ db, int* err)
{
    extern __shared__ __align__(1024) uint8_t sm[];
    __shared__ uint64_t full[MAXSLOT], empty[MAXSLOT], done;
    __shared__ uint32_t tmem_s;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int kx0 = blockIdx.y * p.nkx;
    const int c0 = (int)(blockIdx.z % p.cparts) * p.CB * p.cx, o0 = (int)(blockIdx.z / p.cparts) * p.OB * p.cy;
    const int ca = p.up ? p.cy : p.cx, cn = p.up ? p.cx : p.cy;   // channels per block of the M and N side
    const bool bias = db && blockIdx.y == 0 && blockIdx.z % p.cparts == 0;   // each dy tile counts once
    if (threadIdx.x == 0) {
        for (int q = 0; q < p.stages; q++) {
            mbar_init(&full[q], 1);
            mbar_init(&empty[q], bias ? 1 + EPW : 1);
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
            expect_tx(&full[sl], p.atx + p.bbytes);
            // blocks of `c` channels, nblk of them, from channel f on
            auto box = [&](uint8_t* d, const CUtensorMap* m, int c, int f, int nblk, uint32_t bytes, int x, int y) {
                if (c == 8) tma5(d, m, 0, x, y, f / 8, nb, &full[sl]);
                else
                    for (int k = 0; k < nblk; k++) tma4(d + k * bytes, m, f + k * c, x, y, nb, &full[sl]);
            };
            if (p.up) {
                for (int ab = 0; ab < 4; ab++)
                    box(A + (uint32_t)(ab * p.OB) * p.pitchA, &maps.a[ab], p.cy, o0, p.OB, p.pitchA, x0, y0);
                box(B, &maps.b, p.cx, c0, p.CB, p.pitchB, x0, y0);
            } else {
                box(A, &maps.a[0], p.cx, c0, p.CB, p.jr * p.pitchA, x0 - 1, y0 - 1);
                box(B, &maps.b, p.cy, o0, p.OB, p.rr * p.pitchB, x0, y0);
            }
        }
        for (int k = i > p.stages ? i - p.stages : 0; k < i; k++)
            if (!mbar_wait(&full[k % p.stages], (k / p.stages) & 1)) ok = false;
    } else if (warp == EPW + 1) {        // as in k_conv: the warp runs the loops, one lane issues
        const bool el = elect1();
        const uint32_t idesc = idesc_bf16(p.n) | 1u << 15 | 1u << 16;   // both operands MN-major
        // MN-major: without swizzle LBO steps 8 pixels and SBO to the next chunk plane, with
        // it SBO steps 8 pixels and LBO to the next (block, row) pair.  16-byte units per pixel:
        const uint32_t pa = ca / 8, pn = cn / 8;
        auto desc = [&](int c, uint32_t pitch) {
            return c == 8 ? sdesc(0, 128, pitch) : sdesc(0, pitch, 16 * c) | swizzle_code(c);
        };
        const uint64_t dA = desc(ca, p.pitchA) + (su32(sm) >> 4), dB = desc(cn, p.pitchB) + (su32(sm) >> 4);
        MmaEntry* tab = reinterpret_cast<MmaEntry*>(sm + p.toff);
        const int per = p.nkx * p.mb, n = p.ksteps * per;
        for (int q = lane; q < n; q += 32) {
            const int s = q / per, t = q - s * per, k = t / p.mb, b = t - k * p.mb;
            tab[q] = MmaEntry{(kx0 + k + 16 * s) * pa + (uint32_t)(b * (128 / ca)) * (p.pitchA >> 4),
                              (p.abytes >> 4) + 16 * s * pn | (uint32_t)(t * p.n) << 16};
        }
        __syncwarp();
        int i = 0;
        for (int u = blockIdx.x; u < p.units; u += gridDim.x, i++) {
            const int sl = i % p.stages;
            if (!all_lanes(mbar_wait(&full[sl], (i / p.stages) & 1))) {
                ok = false;
                break;
            }
            tc_fence_after();
            const uint32_t at = (uint32_t)sl * (p.stage >> 4);
            if (el) issue(tab, n, tmem, dA + at, dB + at, idesc, i == 0 ? per : 0);
            if (el) umma_commit(&empty[sl]);
        }
        if (el) umma_commit(&done);
        if (!mbar_wait(&done, 0)) ok = false;
    }
    // bias: these warps wait for the sums anyway and add up dy's staged pixels meanwhile.  A
    // thread sums 8 channels over its pixels, neighbouring threads on neighbouring chunks.
    const int cpb = p.cy / 8, nch = p.OB * cpb, lanes = 32 * EPW / nch;
    const int ch = threadIdx.x % nch, ln = threadIdx.x / nch;
    float bs[8];
#pragma unroll
    for (int e = 0; e < 8; e++) bs[e] = 0.f;
    if (bias && warp < EPW) {
        const uint32_t pitch = p.up ? p.pitchA : p.rr * p.pitchB;    // bytes of a staged block
        const uint32_t px = 2 * p.cy, swz = cpb - 1;                 // SWIZZLE_(2 cy)B: chunk ^ 128-byte line
        const uint32_t from = su32(sm) + (p.up ? 0 : p.abytes) + (ch / cpb) * pitch + (ch % cpb) * 16;
        const int npx = p.rr * p.tw;
        auto load = [&](uint32_t at, float* f) {
            uint4 v;
            at ^= (at >> 7 & swz) << 4;
            asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at));
            unpack8(v, f);
        };
        int i = 0;
        for (int u = blockIdx.x; u < p.units; u += gridDim.x, i++) {
            const int sl = i % p.stages;
            if (!all_lanes(mbar_wait(&full[sl], (i / p.stages) & 1))) {
                ok = false;
                break;
            }
            if (ln < lanes)
                for (int ab = 0; ab < (p.up ? 4 : 1); ab++) {
                    const uint32_t at = from + (uint32_t)sl * p.stage + (uint32_t)(ab * p.OB) * pitch;
                    int q = ln;
                    for (; q + 3 * lanes < npx; q += 4 * lanes) {
                        float f[4][8];
#pragma unroll
                        for (int k = 0; k < 4; k++) load(at + (uint32_t)(q + k * lanes) * px, f[k]);
#pragma unroll
                        for (int e = 0; e < 8; e++) bs[e] += (f[0][e] + f[1][e]) + (f[2][e] + f[3][e]);
                    }
                    for (; q < npx; q += lanes) {
                        float f[8];
                        load(at + (uint32_t)q * px, f);
#pragma unroll
                        for (int e = 0; e < 8; e++) bs[e] += f[e];
                    }
                }
            __syncwarp();
            if (lane == 0) mbar_arrive1(&empty[sl]);
        }
    }
    // TMEM loads are warp-collective and shared memory is reused: the decision is the block's
    const bool all_ok = __syncthreads_and(ok ? 1 : 0) != 0;
    tc_fence_after();
    if (all_ok) {
        const int quad = warp & 3, set = warp >> 2;
        const bool epi = warp < EPW;
        const int row = quad * 32 + lane;
        float* acc = reinterpret_cast<float*>(sm);
        const int cw = p.CB * p.cx, ow = p.OB * p.cy, na = ow * 9 * cw;
        const bool direct = p.up || p.rr == 1;
        // 2x2: lanes are rows of du, so the sums go through shared memory (rows one word apart
        // in banks) to be added along them
        const int ups = cw + 1;
        const bool staged = p.up && p.staged;
        if (bias) {
            if (epi)
#pragma unroll
                for (int e = 0; e < 8; e++) acc[threadIdx.x * 9 + e] = bs[e];
            __syncthreads();
            // channel o of the CTA's 8 nch, one of S partial sums over the pixel lanes
            const int no = 8 * nch, S = max(1, 32 * EPW / no);
            for (int t = threadIdx.x; t < S * no; t += CTHREADS) {
                const int o = t % no;
                float v = 0.f;
                for (int l = t / no; l < lanes; l += S) v += acc[(l * nch + o / 8) * 9 + o % 8];
                if (o0 + o < p.co) atomicAdd(db + o0 + o, v);
            }
            __syncthreads();
        }
        if (!direct) {
            for (int q = threadIdx.x; q < na; q += CTHREADS) acc[q] = 0.f;
            __syncthreads();
        }
        bool nan = false;                // a 3x3 sum is NaN: not added here
        for (int rs = 0; rs < (direct ? 1 : p.rr); rs++) {
            // in shared memory one dy row r at a time: then j - r = ky names every sum once
            if (epi)
                for (int t = set; t < p.nkx * p.mb; t += EPW / 4) {
                    const int k = t / p.mb, b = t - k * p.mb;
                    const int at = b * (128 / ca) + row / ca, ch = row % ca;     // M side: pair, channel
                    const uint32_t td = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(t * p.n);
                    const int kx = kx0 + k;
                    for (int n8 = 0; n8 < p.n; n8 += 8) {
                        const int u = n8 / cn, nc = n8 - u * cn;                  // N side: pair, channel
                        if (!direct && u % p.rr != rs) continue;
                        float v[8];
                        tmem_ld8(td + n8, v);
                        if (at >= p.atoms) continue;
                        if (p.up) {
                            const int ab = at / p.OB, o = o0 + (at - ab * p.OB) * p.cy + ch, c = c0 + u * p.cx + nc;
                            if (staged) {
#pragma unroll
                                for (int q = 0; q < 8; q++) acc[(at * p.cy + ch) * ups + u * p.cx + nc + q] = v[q];
                                continue;
                            }
                            if (o >= p.co || c >= p.ci) continue;
                            float* d = dw + (long long)(ab * p.co + o) * p.ci + c;
#pragma unroll
                            for (int q = 0; q < 8; q++) atomicAdd(d + q, v[q]);
                            continue;
                        }
                        const int cbk = at / p.jr, j = at - cbk * p.jr, ob = u / p.rr, r = u - ob * p.rr;
                        const int ky = j - r;
                        if (ky < 0 || ky > 2 || kx > 2) continue;
                        const int tap = ky * 3 + kx, cl = cbk * p.cx + ch, ol = ob * p.cy + nc;
                        if (direct) {
                            if (c0 + cl >= p.ci || o0 + ol >= p.co) continue;
                            float* d = dw + ((long long)(o0 + ol) * 9 + tap) * p.ci + c0 + cl;
                            const float sum = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
                            if (sum == sum) {        // none of them is NaN
#pragma unroll
                                for (int q = 0; q < 8; q++) atomicAdd(d + (long long)q * 9 * p.ci, v[q]);
                            } else {
                                nan = true;
#pragma unroll
                                for (int q = 0; q < 8; q++)
                                    if (v[q] == v[q]) atomicAdd(d + (long long)q * 9 * p.ci, v[q]);
                            }
                        } else {
#pragma unroll
                            for (int q = 0; q < 8; q++) acc[((ol + q) * 9 + tap) * cw + cl] += v[q];
                        }
                    }
                }
            if (!direct) __syncthreads();
        }
        if (staged) {
            __syncthreads();
            for (int q = threadIdx.x; q < 4 * ow * cw; q += CTHREADS) {
                const int r = q / cw, cl = q - r * cw, ab = r / ow, ol = r - ab * ow;
                if (o0 + ol < p.co && c0 + cl < p.ci)
                    atomicAdd(dw + (long long)(ab * p.co + o0 + ol) * p.ci + c0 + cl, acc[r * ups + cl]);
            }
        }
        if (!direct)
            for (int q = threadIdx.x; q < na; q += CTHREADS) {
                const int c = c0 + q % cw, t = q / cw, tap = t % 9, o = o0 + t / 9;
                if (c < p.ci && o < p.co && tap % 3 >= kx0 && tap % 3 < kx0 + p.nkx) {
                    if (acc[q] == acc[q]) atomicAdd(dw + ((long long)o * 9 + tap) * p.ci + c, acc[q]);
                    else nan = true;
                }
            }
        // the same in every thread of the block
        if (__syncthreads_or(nan)) wgrad_repair(p, src, acc, tmem, dw);
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
            const cuuint32_t* box, int cb = 0)
{
    const CUtensorMapSwizzle sw = cb == 64   ? CU_TENSOR_MAP_SWIZZLE_128B
                                  : cb == 32 ? CU_TENSOR_MAP_SWIZZLE_64B
                                  : cb == 16 ? CU_TENSOR_MAP_SWIZZLE_32B
                                             : CU_TENSOR_MAP_SWIZZLE_NONE;
    const cuuint32_t es[5] = {1, 1, 1, 1, 1};
    auto fn = encoder();
    return fn && fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void*>(base), dims, strides, box, es,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
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
// blocks of cb channels of it
bool map_block(CUtensorMap* m, const Act& a, int step, int dx, int dy, int cb, int bw, int bh)
{
    const cuuint64_t px = (cuuint64_t)a.cs * 2;
    const cuuint64_t dims[4] = {(cuuint64_t)a.c, (cuuint64_t)(a.w / step), (cuuint64_t)(a.h / step), (cuuint64_t)a.nb};
    const cuuint64_t st[3] = {px * step, px * a.w * step, px * a.w * a.h};
    const cuuint32_t box[4] = {(cuuint32_t)cb, (cuuint32_t)bw, (cuuint32_t)bh, 1};
    return encode(m, a.p + ((long long)dy * a.w + dx) * a.cs + a.off, 4, dims, st, box, cb);
}
// rows of K-major weights [N][K]: 64 K with the 128-byte swizzle, or as chunk planes
bool map_w(CUtensorMap* m, const bf16* w, int N, int K, int bn, bool blocks)
{
    if (blocks) {
        const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)N}, st[1] = {(cuuint64_t)K * 2};
        const cuuint32_t box[2] = {64, (cuuint32_t)bn};
        return encode(m, w, 2, dims, st, box, 64);
    }
    const cuuint64_t dims[3] = {8, (cuuint64_t)N, (cuuint64_t)(K / 8)};
    const cuuint64_t st[2] = {(cuuint64_t)K * 2, 16};
    const cuuint32_t box[3] = {8, (cuuint32_t)bn, 2};
    return encode(m, w, 3, dims, st, box);
}

// cycles of a box line of cb channels, and of an M = 128 MMA of n columns (measured alone)
double line_cost(int cb) { return cb == 64 ? 7.0 : cb == 32 ? 3.4 : cb == 16 ? 2.7 : 1.6; }
double mma_cost(int n) { return std::max(40.0, 32 + n / 4.0); }

// Tiles of a convolution over an nb x h x w output grid with N output channels and, per
// map, C input channels.  Columns: 128 at a time where the width is a multiple of 128
// (one MMA block per row); else whole rows (up to 254) one after the other in the MMA's
// 128 positions; else 126.  The number of rows ro, the output channels bn per CTA and
// whether the weights stay resident are chosen by a cost in cycles: staged lines, MMA
// time, epilogue, and waves of persistent CTAs.  Chunk planes are left to
// channel counts that are no multiple of 16 and to weights that do not fit.
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
    p.pair8 = three && C == 8;
    const int K = (three ? 9 : nmap) * C;
    const bool want_tap = three && (w % 128 != 0 || C % 16 != 0);
    const int n16 = up_to(N, 16);
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
        p.rows = ro + 2 * p.halo;
        p.mstep = rowmode ? p.wp : 128;
        p.nblk = rowmode ? ro : div_up((long long)(ro - 1) * p.wp + p.txw, 128);
        p.ty = div_up(h, ro);
        if ((long long)p.tx * p.ty * nb > 0x7fffffff) continue;
        p.tiles = p.tx * p.ty * nb;
        // mode 0: swizzled blocks, weights resident; 1, 2: chunk planes, weights resident / streamed
        for (int mode = 0; mode < 3; mode++) {
            if (mode == 0 ? C % 16 != 0 : mode == 2 && p.pair8) continue;
            p.stream = mode == 2;
            p.cb = mode ? 0 : C > 32 ? 64 : C > 16 ? 32 : 16;
            p.pitch = mode ? 16 : 2 * p.cb;
            p.nch = p.pair8 ? 1 : 2;
            p.B = p.cb ? div_up(C, p.cb) : div_up(C, 16);
            p.taps = three ? (p.pair8 ? 5 : 9) : 1;
            p.plane = (uint32_t)(p.rows * p.wp) * p.pitch;
            p.abytes = p.cb ? p.plane : p.nch * p.plane;
            p.zeros = p.pair8 ? up_to(p.abytes, 128) : 0;
            p.aslot = up_to(p.pair8 ? p.zeros + ZEROS : p.abytes, 1024);
            const int BB = p.B * nmap, lines = p.rows * p.wp * (p.cb ? 1 : p.nch);
            // the last block of positions may read past the last plane: keep that in bounds
            const int last = (p.nblk - 1) * p.mstep + 127 + (three ? 2 * p.wp + 2 : 0);
            const int over = std::max(0, last + 1 - p.rows * p.wp) * (int)p.pitch;
            for (int parts = 1; parts <= n16 / 16; parts++) {
                const int bn = up_to(div_up(n16, parts), 16);
                if (bn > 128 || p.nblk * bn > 512 || (parts > 1 && bn == up_to(div_up(n16, parts - 1), 16))) continue;
                p.bn = bn;
                p.wtap = 32u * bn;
                p.nbuf = 2 * p.nblk * bn <= 512 ? 2 : 1;
                p.tcols = tmem_cols(p.nbuf * p.nblk * bn);
                p.wbytes = p.stream ? 0 : p.cb ? 128u * bn * div_up(K, 64) : (uint32_t)(BB * p.taps) * p.wtap;
                p.slot = p.aslot + (p.stream ? p.taps * p.wtap : 0);
                p.groups = p.stream ? 1 : p.cb ? nmap * C / 16 : BB;
                p.entries = p.groups * p.taps * p.nblk;
                const size_t rest = p.wbytes + over + up_to(8 * p.entries, 128);
                if (rest + 2 * (size_t)p.slot > SMEM_MAX) continue;
                int slots = (int)std::min<size_t>(MAXSLOT, (SMEM_MAX - rest) / p.slot);
                p.tapmajor = want_tap && BB <= slots && !p.stream;
                p.slots = slots = std::min(slots, std::max(2, 3 * BB));
                const int split = div_up(n16, bn), per = std::max(1, SMS / split);
                const int waves = div_up(p.tiles, std::min(per, p.tiles));
                const double load = (double)BB * (lines * line_cost(p.cb) + (p.stream ? p.taps * 2 * bn * 1.6 : 0));
                const double mma = (double)(p.cb ? nmap * C / 16 : BB) * p.taps * p.nblk * mma_cost(bn);
                const double epi = div_up(p.nblk, 4) * (bn / 8) * 60.0 + 200;
                const bool ahead = slots >= (p.tapmajor ? 2 * BB : 2);
                const double body = std::max(epi, ahead ? std::max(load, mma) : load + mma);
                const double tile = (p.nbuf == 2 ? body : std::max(load, mma + epi)) + 150;
                const double wload = p.wbytes / (p.cb ? 128.0 : 16.0) * line_cost(p.cb ? 64 : 8);
                const double cost = waves * tile + load + mma + epi + 2500 + wload + (want_tap && !p.tapmajor ? 1e9 : 0);
                if (cost < best_cost) {
                    best_cost = cost;
                    p.woff = (uint32_t)p.slots * p.slot;
                    p.toff = p.woff + p.wbytes;
                    best = p;
                    smem = (size_t)p.slots * p.slot + rest;
                    gx = std::min(per, p.tiles);
                    gy = split;
                }
            }
        }
    }
    return best_cost < 1e299;
}

// The plans are pure functions of a layer's sizes, about 10 us of search each: the last few
// are kept per thread (direct-mapped by a hash of the sizes, bounded).
template <class T, int NKEY>
struct PlanCache {
    struct Slot {
        int key[NKEY];
        bool ok, set = false;
        T plan;
    };
    Slot slots[64];
    Slot& at(const int* key, bool& hit)
    {
        uint32_t h = 2166136261u;
        for (int q = 0; q < NKEY; q++) h = (h ^ (uint32_t)key[q]) * 16777619u;
        Slot& s = slots[(h ^ h >> 15) & 63];
        hit = s.set && std::equal(key, key + NKEY, s.key);
        if (!hit) {
            std::copy(key, key + NKEY, s.key);
            s.set = true;
        }
        return s;
    }
};

template <class EP>
cudaError_t conv_launch(const Act* x, int nmap, int step, const bf16* w, int K, int nb, int h, int wd, int N, bool three,
                        const EP& ep, int* err, cudaStream_t st)
{
    struct Plan {
        ConvP p;
        size_t smem;
        int gx, gy;
    };
    static thread_local PlanCache<Plan, 7> cache;
    const int key[7] = {nb, h, wd, N, x->c, nmap, three};
    bool hit;
    auto& slot = cache.at(key, hit);
    if (!hit) slot.ok = conv_plan(slot.plan.p, slot.plan.smem, slot.plan.gx, slot.plan.gy, nb, h, wd, N, x->c, nmap, three);
    if (!slot.ok) return cudaErrorInvalidValue;
    const ConvP& p = slot.plan.p;
    const size_t smem = slot.plan.smem;
    const int gx = slot.plan.gx, gy = slot.plan.gy;
    ConvMaps maps;
    for (int q = 0; q < nmap; q++)
        if (!(p.cb ? map_block(&maps.x[q], *x, step, q & 1, q >> 1, p.cb, p.wp, p.rows)
                   : map_act(&maps.x[q], *x, step, q & 1, q >> 1, p.wp, p.rows, p.nch)))
            return cudaErrorInvalidValue;
    for (int q = nmap; q < 4; q++) maps.x[q] = maps.x[0];
    if (!map_w(&maps.w, w, N, K, p.bn, p.cb != 0)) return cudaErrorInvalidValue;
    static unsigned long long opted = 0;
    const cudaError_t e = ertm::smem_opt_in(k_conv<EP>, SMEM_MAX, &opted);
    if (e != cudaSuccess) return e;
    return ertm::launch_pdl(k_conv<EP>, dim3(gx, gy), dim3(CTHREADS), smem, st, maps, p, ep, err);
}

// Tiles of a weight gradient.  3x3: rr rows of dy against rr + 2 of x; more rows re-read
// less of x and waste fewer row pairs but need TMEM (mb * n columns per kx, 512 in all)
// and shared memory for two stages or more.  At most `most` CTAs add to an element of dw;
// with one the sum is repeatable.
bool wgrad_plan(WgP& best, size_t& smem, dim3& grid, int nb, int h, int w, int ci, int co, bool up, int most)
{
    WgP p{};
    p.nb = nb;
    p.h = h;
    p.w = w;
    p.ci = ci;
    p.co = co;
    p.up = up;
    auto block = [](int c) { return c % 16 ? 8 : c > 32 ? 64 : c > 16 ? 32 : 16; };
    p.cx = block(ci);
    p.cy = block(co);
    const int cblk = div_up(ci, p.cx), oblk = div_up(co, p.cy);
    const int ca = up ? p.cy : p.cx, cn = up ? p.cx : p.cy;
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
                for (int cdiv = 1; cdiv < 2 * cblk; cdiv *= 2)   // down to one block
                    for (int odiv = 1; odiv < 2 * oblk; odiv *= 2) {
                        p.CB = div_up(cblk, cdiv);
                        p.OB = div_up(oblk, odiv);
                        double load;
                        if (up) {
                            if (p.cx == 8 && p.CB % 2) p.CB++;          // N in multiples of 16
                            p.jr = rr;
                            p.atoms = 4 * p.OB;
                            p.n = p.cx * p.CB;
                            p.pitchA = (uint32_t)(rr * tw * 2 * ca);
                            p.pitchB = (uint32_t)(rr * tw * 2 * cn);
                            p.ksteps = rr * tw / 16;
                            p.atx = (uint32_t)p.atoms * p.pitchA;
                            p.bbytes = (uint32_t)p.CB * p.pitchB;
                            load = (p.atoms * line_cost(ca) + p.CB * line_cost(cn)) * rr * tw;
                        } else {
                            if (p.cy == 8 && (p.OB * rr) % 2) p.OB++;
                            p.jr = rr + 2;
                            p.atoms = p.CB * p.jr;
                            p.n = p.cy * p.OB * rr;
                            p.pitchA = (uint32_t)((tw + 2) * 2 * ca);
                            p.pitchB = (uint32_t)(tw * 2 * cn);
                            p.ksteps = tw / 16;
                            p.atx = (uint32_t)p.atoms * p.pitchA;
                            p.bbytes = (uint32_t)(p.OB * rr) * p.pitchB;
                            load = p.atoms * (tw + 2) * line_cost(ca) + p.OB * rr * tw * line_cost(cn);
                            // swizzled boxes start on their repeat: one block, or whole repeats between blocks
                            if (p.cx > 8 && p.CB > 1 && (p.jr * p.pitchA) % 1024) continue;
                            if (p.cy > 8 && p.OB > 1 && (rr * p.pitchB) % 1024) continue;
                        }
                        if (up && ((ca > 8 && p.pitchA % 1024) || (cn > 8 && p.CB > 1 && p.pitchB % 1024))) continue;
                        p.abytes = up_to(p.atx, 1024);
                        const int per128 = 128 / ca;
                        p.mb = div_up(p.atoms, per128);
                        const int cols = p.mb * p.nkx * p.n;
                        if (p.n > 256 || cols > 512 || p.CB > 256 || p.OB > 256 || p.pitchA > 262000 || p.pitchB > 262000)
                            continue;
                        p.stage = up_to(p.abytes + p.bbytes, 1024);
                        // MMA blocks are 128 channels: the last may read past the staged ones
                        const int over = std::max(0, (int)(p.mb * per128 - p.atoms) * (int)p.pitchA + 8 * ca - (int)p.bbytes);
                        const int table = up_to(8 * p.ksteps * p.nkx * p.mb, 128);
                        if (2 * (size_t)p.stage + over + table > SMEM_MAX) continue;
                        const int stages = std::min(8, (int)((SMEM_MAX - over - table) / p.stage));
                        size_t accb = up    ? (size_t)4 * p.OB * p.cy * (p.CB * p.cx + 1) * 4
                                      : rr == 1 ? 0
                                                : (size_t)p.OB * p.cy * 9 * p.CB * p.cx * 4;
                        p.staged = up && accb <= SMEM_MAX;
                        if (up && !p.staged) accb = 0;
                        if (accb > SMEM_MAX) continue;
                        p.stages = stages;
                        p.tcols = tmem_cols(cols);
                        p.cparts = div_up(cblk, p.CB);
                        const int others = p.kgroups * p.cparts * div_up(oblk, p.OB);
                        const int px = up ? rr * tw : tw;        // accumulator chain per unit
                        const int least = div_up((long long)p.units * px, 4096);
                        const int splits = std::min({p.units, most, std::max(std::max(1, SMS / others), least)});
                        const int waves = div_up((long long)splits * others, SMS);
                        const double mma = (double)p.ksteps * p.nkx * p.mb * mma_cost(p.n);
                        const double sums = up ? (double)p.mb * 128 * p.n : 9.0 * p.CB * p.cx * p.OB * p.cy * p.nkx / 3 * rr;
                        const double epi = 3000 + sums / (p.up && !p.staged ? 2 : 16) + (double)cols * 2 * (up ? 1 : std::min(rr, 4));
                        const double cost = waves * (div_up(p.units, splits) * (std::max(load, mma) + 250) + load + epi);
                        if (cost < best_cost) {
                            best_cost = cost;
                            best = p;
                            best.toff = (uint32_t)stages * p.stage;
                            // the bias's partial sums take 36 bytes of every summing thread
                            smem = std::max({(size_t)stages * p.stage + over + table, accb, (size_t)32 * EPW * 36});
                            grid = dim3(splits, p.kgroups, p.cparts * div_up(oblk, p.OB));
                        }
                    }
            }
        }
    }
    return best_cost < 1e299;
}

cudaError_t wgrad_launch(const Act& x, const Act& dy, float* dw, float* db, bool up, int most, int* err, cudaStream_t st)
{
    struct Plan {
        WgP p;
        size_t smem;
        dim3 grid;
    };
    most = std::max(1, most);
    static thread_local PlanCache<Plan, 7> cache;
    const int key[7] = {x.nb, x.h, x.w, x.c, dy.c, up, most};
    bool hit;
    auto& slot = cache.at(key, hit);
    if (!hit) slot.ok = wgrad_plan(slot.plan.p, slot.plan.smem, slot.plan.grid, x.nb, x.h, x.w, x.c, dy.c, up, most);
    if (!slot.ok) return cudaErrorInvalidValue;
    const WgP& p = slot.plan.p;
    const size_t smem = slot.plan.smem;
    const dim3 grid = slot.plan.grid;
    WgMaps maps;
    auto map = [](CUtensorMap* m, const Act& a, int step, int q, int c, int bw, int bh, int n) {
        return c == 8 ? map_act(m, a, step, q & 1, q >> 1, bw, bh, n) : map_block(m, a, step, q & 1, q >> 1, c, bw, bh);
    };
    bool ok = true;
    if (up) {
        for (int q = 0; q < 4; q++) ok = ok && map(&maps.a[q], dy, 2, q, p.cy, p.tw, p.rr, p.OB);
        ok = ok && map(&maps.b, x, 1, 0, p.cx, p.tw, p.rr, p.CB);
    } else {
        ok = map(&maps.a[0], x, 1, 0, p.cx, p.tw + 2, p.jr, p.CB);
        for (int q = 1; q < 4; q++) maps.a[q] = maps.a[0];
        ok = ok && map(&maps.b, dy, 1, 0, p.cy, p.tw, p.rr, p.OB);
    }
    if (!ok) return cudaErrorInvalidValue;
    static unsigned long long opted = 0;
    const cudaError_t e = ertm::smem_opt_in(k_wgrad, SMEM_MAX, &opted);
    if (e != cudaSuccess) return e;
    return ertm::launch_pdl(k_wgrad, grid, dim3(CTHREADS), smem, st, maps, p, WgSrc{x, dy}, dw, db, err);
}

}  // namespace

namespace ertm {
int nn_conv3x3_wgrad(const ertm_nn_act* x, const ertm_nn_act* dy, float* dw, float* db, int splitk, int* err,
                     void* stream)
{
    if (!act_ok(x) || !act_ok(dy) || !dw || (db && !same_grid(x, dy))) return ERTM_EINVAL;
    Act da = act_of(dy);            // dy's pixels are taken in x's grid, in order
    da.nb = x->n;
    da.h = x->h;
    da.w = x->w;
    return rc_of(wgrad_launch(act_of(x), da, dw, db, false, splitk, err, (cudaStream_t)stream));
}

int nn_up2_wgrad(const ertm_nn_act* x, const ertm_nn_act* dy, float* du, float* db, int splitk, int* err, void* stream)
{
    if (!act_ok(x) || !act_ok(dy) || !du || dy->h != 2 * x->h || dy->w != 2 * x->w || (db && dy->n != x->n))
        return ERTM_EINVAL;
    Act da = act_of(dy);
    da.nb = x->n;
    return rc_of(wgrad_launch(act_of(x), da, du, db, true, splitk, err, (cudaStream_t)stream));
}
}  // namespace ertm

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
    return ertm::nn_conv3x3_wgrad(x, dy, dw, nullptr, splitk, err, stream);
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
    return ertm::nn_up2_wgrad(x, dy, du, nullptr, splitk, err, stream);
}

}  // extern "C"
