// Learned LSRTM preconditioner: the plain GEMM on the tensor cores and the U-Net's
// elementwise kernels (the convolutions are in nn_conv.cu).
//
//   D[M x N] = sum_k A[m, k] B[n, k]          (A, B BF16; D FP32 in TMEM)
// issued with tcgen05.mma (kind::f16, M = 128 rows per CTA, N = BN <= 128
// columns, K = 16 per instruction) by one thread of the CTA.  All 128 threads stage
// the operands in shared memory, 8 consecutive K elements (16 bytes) of one row at a
// time, into a ring of 3-4 stages with cp.async (zero-fill past the bounds),
// several K tiles ahead of the tensor core; tcgen05.commit on a per-stage mbarrier
// tells them when a stage may be refilled.  After the K loop each warp reads its 32
// accumulator rows from TMEM (tcgen05.ld 32x32b).
//
// Shared-memory operand layout (K-major, no swizzle): element (r, k) of an
// R-row, 64-column stage at byte ((k / 8) * R + r) * 16 + (k % 8) * 2, i.e. the
// 8 x 16-byte core matrices of the canonical layout with SBO = 128 bytes
// (next 8 rows) and LBO = R * 16 bytes (next 8 K elements).
#include <algorithm>

#include "nn_common.cuh"

namespace {

constexpr int BK = 64;       // K elements per stage
constexpr int NT = 128;      // threads per CTA

// rows of a K-major matrix [rows][ld]: address of 8 consecutive K elements of row r from
// k on (k % 8 == 0), or nullptr past the bounds
struct LoadRows {
    const bf16* p;
    int rows, K, ld;
    __device__ __forceinline__ const bf16* src(int r, int k) const
    {
        if (r >= rows || k >= K) return nullptr;
        return p + (long long)r * ld + k;
    }
};

// FP32 output, 8 consecutive columns n0..n0+7 of row m
struct EpiF32 {
    float* y;
    int cs, N, M;
    __device__ __forceinline__ void operator()(int m, int n0, const float* v) const
    {
        if (m >= M) return;
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const int n = n0 + q;
            if (n >= N) break;
            y[(long long)m * cs + n] = v[q];
        }
    }
};

// ---------------------------------------------------------------------------
// The GEMM kernel
// ---------------------------------------------------------------------------
// ring depth: four stages up to BN = 64 (up to 72 KB), three at BN = 128 (96 KB)
template <int BN>
struct Ring {
    static constexpr int N = BN >= 128 ? 3 : 4;
};
template <int BN>
struct Smem {
    static constexpr int NS = Ring<BN>::N;
    alignas(128) uint8_t a[NS][BM * BK * 2];
    alignas(128) uint8_t b[NS][BN * BK * 2];
    uint64_t bar[NS];
    uint32_t tmem;
};

__device__ __forceinline__ void cp16(void* sdst, const void* gsrc)
{
    // 16 bytes global -> shared, asynchronous; a null source zero-fills
    const uint32_t n = gsrc ? 16u : 0u;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(su32(sdst)),
                 "l"(gsrc ? gsrc : sdst), "r"(n)
                 : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// stage one operand tile: rows [r0, r0 + R), K chunk [k0, k0 + 64)
template <int R, class L>
__device__ __forceinline__ void stage(uint8_t* dst, const L& ld, int r0, int k0)
{
    constexpr int CH = R * (BK / 8);   // 16-byte chunks
    // chunk = 8 K elements of one row; core matrix (8 rows x 16 B)
#pragma unroll 4
    for (int q = threadIdx.x; q < CH; q += NT) {
        const int r = q % R, j = q / R;    // consecutive threads take consecutive rows
        cp16(dst + ((size_t)j * R + r) * 16, ld.src(r0 + r, k0 + j * 8));
    }
}

template <int BN, class LA, class LB, class EP>
__global__ void __launch_bounds__(NT) k_gemm(LA la, LB lb, EP ep, int M, int N, int K, int* err)
{
    extern __shared__ __align__(128) uint8_t smraw[];
    Smem<BN>& S = *reinterpret_cast<Smem<BN>*>(smraw);
    constexpr int TCOLS = BN < 32 ? 32 : BN;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;

    constexpr int NS = Smem<BN>::NS;
    if (threadIdx.x == 0) {
        for (int q = 0; q < NS; q++) mbar_init(&S.bar[q], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(&S.tmem)),
                     "r"(TCOLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = S.tmem;
    constexpr uint32_t IDESC = idesc_bf16(BN);
    bool ok = true;
    const int nu = (K + BK - 1) / BK;
    // every thread copies its chunks of K tile u into slot u % NS with cp.async, one
    // commit group per tile (empty groups keep the count uniform)
    auto issue = [&](int u) {
        if (u < nu) {
            const int sl = u % NS;
            stage<BM>(S.a[sl], la, m0, u * BK);
            stage<BN>(S.b[sl], lb, n0, u * BK);
        }
        cp_commit();
    };
    for (int u = 0; u < NS - 1; u++) issue(u);
    for (int u = 0; u < nu; ++u) {
        cp_wait<NS - 2>();        // this thread's copies of tile u have landed
        proxy_fence();            // ... and are visible to the tensor core's async proxy
        __syncthreads();          // ... for every thread's chunks
        const int sl = u % NS;
        if (threadIdx.x == 0 && ok) {
            tc_fence_after();
            const uint32_t a0 = su32(S.a[sl]), b0 = su32(S.b[sl]);
#pragma unroll
            for (int j = 0; j < BK / 16; j++) {
                // K step j covers the core-matrix columns 2j, 2j+1
                const uint64_t da = sdesc(a0 + (uint32_t)(2 * j * BM * 16), BM * 16);
                const uint64_t db = sdesc(b0 + (uint32_t)(2 * j * BN * 16), BN * 16);
                umma(tmem, da, db, IDESC, (u > 0 || j > 0) ? 1u : 0u);
            }
            umma_commit(&S.bar[sl]);
        }
        // refill slot (u - 1) % NS with tile u + NS - 1 once tile u-1's MMAs read it
        const int un = u + NS - 1;
        if (un < nu && u >= 1 && ok) ok = mbar_wait(&S.bar[(u - 1) % NS], ((u - 1) / NS) & 1);
        issue(ok ? un : nu);
    }
    cp_wait<0>();
    if (nu > 0 && ok) ok = mbar_wait(&S.bar[(nu - 1) % NS], ((nu - 1) / NS) & 1);
    // the other stage's last commit precedes it, so every MMA has completed;
    // the TMEM loads below are warp-collective, so the decision is block-uniform
    const bool all_ok = __syncthreads_and(ok ? 1 : 0) != 0;
    tc_fence_after();
    if (nu > 0 && all_ok) {
        const int m = m0 + warp * 32 + lane;
        const uint32_t trow = tmem + ((uint32_t)(warp * 32) << 16);
#pragma unroll 1
        for (int c = 0; c < BN; c += 8) {
            float v[8];
            tmem_ld8(trow + c, v);
            ep(m, n0 + c, v);
        }
    }
    if (!ok && err) atomicExch(err, NN_WAIT);
    tc_fence_before();
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TCOLS) : "memory");
}

template <int BN, class LA, class LB, class EP>
cudaError_t gemm_bn(const LA& la, const LB& lb, const EP& ep, int M, int N, int K, int* err, cudaStream_t st)
{
    const size_t smem = sizeof(Smem<BN>);
    static unsigned long long opted = 0;   // devices with the opt-in made
    cudaError_t attr = ertm::smem_opt_in(k_gemm<BN, LA, LB, EP>, smem, &opted);
    if (attr != cudaSuccess) return attr;
    dim3 grid((M + BM - 1) / BM, (N + BN - 1) / BN);
    k_gemm<BN, LA, LB, EP><<<grid, NT, smem, st>>>(la, lb, ep, M, N, K, err);
    return cudaGetLastError();
}

// N tile: 16 <= BN <= 128, multiple of 16 (tcgen05 M = 128 needs N % 16 == 0)
template <class LA, class LB, class EP>
cudaError_t gemm(const LA& la, const LB& lb, const EP& ep, int M, int N, int K, int* err, cudaStream_t st)
{
    if (N <= 16) return gemm_bn<16>(la, lb, ep, M, N, K, err, st);
    if (N <= 32) return gemm_bn<32>(la, lb, ep, M, N, K, err, st);
    if (N <= 64) return gemm_bn<64>(la, lb, ep, M, N, K, err, st);
    return gemm_bn<128>(la, lb, ep, M, N, K, err, st);
}

// ---------------------------------------------------------------------------
// Elementwise kernels
// ---------------------------------------------------------------------------
// 2x2 max pooling of an NHWC view into a dense NHWC output with C channels
__global__ void k_pool_fwd(Act x, bf16* y, long long n)
{
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        const int c = (int)(q % x.c);
        long long t = q / x.c;
        const int j = (int)(t % (x.w / 2));
        t /= (x.w / 2);
        const int i = (int)(t % (x.h / 2)), nb = (int)(t / (x.h / 2));
        float m = -3.0e38f;
        for (int a = 0; a < 2; a++)
            for (int b = 0; b < 2; b++)
                m = fmaxf(m, __bfloat162float(x.p[((long long)(nb * x.h + 2 * i + a) * x.w + 2 * j + b) * x.cs + x.off + c]));
        y[q] = __float2bfloat16(m);
    }
}

// max pooling backward: the gradient goes to the first maximum of each 2x2 window;
// adds into dx (NHWC view), masked by the ReLU of x when mask != 0
__global__ void k_pool_bwd(Act x, const bf16* dy, bf16* dx, long long n, int mask)
{
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        const int c = (int)(q % x.c);
        long long t = q / x.c;
        const int j = (int)(t % (x.w / 2));
        t /= (x.w / 2);
        const int i = (int)(t % (x.h / 2)), nb = (int)(t / (x.h / 2));
        float m = -3.0e38f;
        long long best = -1;
        for (int a = 0; a < 2; a++)
            for (int b = 0; b < 2; b++) {
                const long long e = ((long long)(nb * x.h + 2 * i + a) * x.w + 2 * j + b) * x.cs + x.off + c;
                const float v = __bfloat162float(x.p[e]);
                if (v > m) { m = v; best = e; }
            }
        const float g = __bfloat162float(dy[q]);
        if (best >= 0 && (!mask || m > 0.f)) dx[best] = __float2bfloat16(__bfloat162float(dx[best]) + g);
    }
}

// The same two with one thread per 8 channels (16-byte accesses): the scalar kernels
// above remain for a pooled tensor off a 16-byte boundary.
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
// pooled pixel (blockIdx.y = image row of the output, over all images) and chunk
__global__ void k_pool_fwd8(Act x, uint4* y)
{
    const int cc = x.c / 8, lw = x.w / 2, n = lw * cc;
    const int row = blockIdx.y, nb = row / (x.h / 2), i = row - nb * (x.h / 2);
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
        const int j = q / cc, c = q - j * cc;
        const bf16* p = x.p + ((long long)(nb * x.h + 2 * i) * x.w + 2 * j) * x.cs + x.off + 8 * c;
        float m[8];
#pragma unroll
        for (int e = 0; e < 8; e++) m[e] = -3.0e38f;
        uint4 u[4];
#pragma unroll
        for (int a = 0; a < 4; a++)
            u[a] = __ldg(reinterpret_cast<const uint4*>(p + ((long long)(a >> 1) * x.w + (a & 1)) * x.cs));
#pragma unroll
        for (int a = 0; a < 4; a++) {
            float f[8];
            unpack8(u[a], f);
#pragma unroll
            for (int e = 0; e < 8; e++) m[e] = fmaxf(m[e], f[e]);
        }
        y[(long long)row * n + q] = pack8(m);
    }
}
__global__ void k_pool_bwd8(Act x, const uint4* __restrict__ dy, bf16* dx, int mask)
{
    const int cc = x.c / 8, lw = x.w / 2, n = lw * cc;
    const int row = blockIdx.y, nb = row / (x.h / 2), i = row - nb * (x.h / 2);
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
        const int j = q / cc, c = q - j * cc;
        const long long at = ((long long)(nb * x.h + 2 * i) * x.w + 2 * j) * x.cs + x.off + 8 * c;
        uint4 u[4], d[4];
        const uint4 gu = __ldg(dy + (long long)row * n + q);
#pragma unroll
        for (int a = 0; a < 4; a++) {
            const long long o = at + ((long long)(a >> 1) * x.w + (a & 1)) * x.cs;
            u[a] = __ldg(reinterpret_cast<const uint4*>(x.p + o));
            d[a] = *reinterpret_cast<const uint4*>(dx + o);
        }
        float m[8], g[8], f[4][8];
        int best[8];
        unpack8(gu, g);
#pragma unroll
        for (int e = 0; e < 8; e++) {
            m[e] = -3.0e38f;
            best[e] = -1;
        }
#pragma unroll
        for (int a = 0; a < 4; a++) {
            unpack8(u[a], f[a]);
#pragma unroll
            for (int e = 0; e < 8; e++)
                if (f[a][e] > m[e]) { m[e] = f[a][e]; best[e] = a; }
        }
#pragma unroll
        for (int a = 0; a < 4; a++) {
            float t[8];
            bool any = false;
            unpack8(d[a], t);
#pragma unroll
            for (int e = 0; e < 8; e++)
                if (best[e] == a && (!mask || m[e] > 0.f)) {
                    t[e] += g[e];
                    any = true;
                }
            if (any) *reinterpret_cast<uint4*>(dx + at + ((long long)(a >> 1) * x.w + (a & 1)) * x.cs) = pack8(t);
        }
    }
}

// bias gradient: db[o] += sum over pixels of dy[p][off + o].  A thread sums 8 channels
// (16-byte loads, neighbouring threads on neighbouring chunks of a pixel) over its
// pixels; blockIdx.y is a block of 32 chunks.
__global__ void __launch_bounds__(256) k_bias_grad(Act dy, long long P, float* db)
{
    __shared__ float part[256 * 9];
    const int cb = min(32, dy.c / 8 - 32 * (int)blockIdx.y), lanes = 256 / cb;
    const int t = threadIdx.x, ch = t % cb, ln = t / cb;
    float s[8];
#pragma unroll
    for (int e = 0; e < 8; e++) s[e] = 0.f;
    if (ln < lanes) {
        const bf16* p = dy.p + dy.off + 8 * (32 * (int)blockIdx.y + ch);
        const long long step = (long long)gridDim.x * lanes;
        long long q = (long long)blockIdx.x * lanes + ln;
        for (; q + 3 * step < P; q += 4 * step) {
            uint4 u[4];
#pragma unroll
            for (int k = 0; k < 4; k++) u[k] = __ldg(reinterpret_cast<const uint4*>(p + (q + k * step) * dy.cs));
#pragma unroll
            for (int k = 0; k < 4; k++) {
                float f[8];
                unpack8(u[k], f);
#pragma unroll
                for (int e = 0; e < 8; e++) s[e] += f[e];
            }
        }
        for (; q < P; q += step) {
            float f[8];
            unpack8(__ldg(reinterpret_cast<const uint4*>(p + q * dy.cs)), f);
#pragma unroll
            for (int e = 0; e < 8; e++) s[e] += f[e];
        }
    }
#pragma unroll
    for (int e = 0; e < 8; e++) part[t * 9 + e] = s[e];
    __syncthreads();
    // channel o of the block's 8 cb, one of S partial sums over the pixel lanes
    const int no = 8 * cb, S = 256 / no, o = t % no, sp = t / no;
    float v = 0.f;
    if (sp < S)
        for (int l = sp; l < lanes; l += S) v += part[(l * cb + o / 8) * 9 + o % 8];
    __syncthreads();
    part[t] = v;
    __syncthreads();
    if (t < no) {
        for (int k = 1; k < S; k++) v += part[k * no + t];
        atomicAdd(db + 256 * blockIdx.y + t, v);
    }
}

// mean-squared-error gradient of an FP32 NHWC output against a target, first C
// channels of cs: g = scale (y - t) (BF16, cs channels, zero in the padding);
// loss += sum (y - t)^2.  One thread per 8 channels, one atomic per block.
__global__ void __launch_bounds__(256) k_mse(const float* __restrict__ y, const float* __restrict__ t, int cs, int C,
                                             long long P, float scale, bf16* __restrict__ g, float* loss, int vec)
{
    const int cc = cs / 8;
    float acc = 0.f;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < P * cc; q += (long long)gridDim.x * blockDim.x) {
        const long long p = cc == 1 ? q : cc == 2 ? q >> 1 : q / cc;
        const int c0 = 8 * (int)(q - p * cc);
        float d[8];
#pragma unroll
        for (int e = 0; e < 8; e++) {
            d[e] = 0.f;
            if (c0 + e < C) {
                const float v = y[p * cs + c0 + e] - t[p * C + c0 + e];
                acc += v * v;
                d[e] = scale * v;
            }
        }
        if (vec) *reinterpret_cast<uint4*>(g + p * cs + c0) = pack8(d);
        else
#pragma unroll
            for (int e = 0; e < 8; e++) g[p * cs + c0 + e] = __float2bfloat16(d[e]);
    }
    for (int k = 16; k; k >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, k);
    __shared__ float part[8];
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        float v = 0.f;
        for (int w = 0; w < 8; w++) v += part[w];
        atomicAdd(loss, v);
    }
}

// Adam on FP32 master weights; writes the BF16 copy used by the GEMMs
__global__ void k_adam(float* w, const float* g, float* m, float* v, bf16* wb, long long n, float lr, float b1,
                       float b2, float eps, float c1, float c2)
{
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        const float gq = g[q];
        const float mq = b1 * m[q] + (1.f - b1) * gq;
        const float vq = b2 * v[q] + (1.f - b2) * gq * gq;
        m[q] = mq;
        v[q] = vq;
        const float wq = w[q] - lr * (mq / c1) / (sqrtf(vq / c2) + eps);
        w[q] = wq;
        wb[q] = __float2bfloat16(wq);
    }
}

// weight re-layouts for the input gradients:
//  conv3: W[o][tap][c] (K = 9 Ci) -> Wf[c][8 - tap][o] (K = 9 Co)
//  up2:   U[(a*2+b)*Co + o][c] (K = Ci) -> Ut[c][(a*2+b)*Co + o] (K = 4 Co)
__global__ void k_flip3(const bf16* w, bf16* wf, int co, int ci)
{
    const long long n = (long long)co * 9 * ci;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        const int c = (int)(q % ci), tap = (int)((q / ci) % 9), o = (int)(q / (9LL * ci));
        wf[((long long)c * 9 + (8 - tap)) * co + o] = w[q];
    }
}
__global__ void k_transpose(const bf16* a, bf16* t, int rows, int cols)
{
    const long long n = (long long)rows * cols;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        const int c = (int)(q % cols), r = (int)(q / cols);
        t[(long long)c * rows + r] = a[q];
    }
}
__global__ void k_f32_to_bf16(const float* a, bf16* b, long long n)
{
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x)
        b[q] = __float2bfloat16(a[q]);
}

// c FP32 values per pixel -> 8 BF16 channels, zero in the padding: one 16-byte store per pixel
__global__ void __launch_bounds__(256) k_pack8(const float* __restrict__ x, uint4* __restrict__ y, int c, long long n)
{
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        float f[8];
#pragma unroll
        for (int e = 0; e < 8; e++) f[e] = e < c ? __ldg(x + q * c + e) : 0.f;
        y[q] = pack8(f);
    }
}

int grid_of(long long n) { return (int)((n + 255) / 256 < 148 * 16 ? (n + 255) / 256 : 148 * 16); }

}  // namespace

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
extern "C" {

int ertm_nn_gemm(const void* a, const void* b, float* d, int M, int N, int K, int* err, void* stream)
{
    if (!aligned16(a) || !aligned16(b) || !d || M < 1 || N < 1 || K < 1 || K % 8) return ERTM_EINVAL;
    LoadRows la{reinterpret_cast<const bf16*>(a), M, K, K};
    LoadRows lb{reinterpret_cast<const bf16*>(b), N, K, K};
    EpiF32 ep{d, N, N, M};
    return rc_of(gemm(la, lb, ep, M, N, K, err, (cudaStream_t)stream));
}

int ertm_nn_pool2(const ertm_nn_act* x, void* y, void* stream)
{
    if (!act_ok(x) || !y || x->h % 2 || x->w % 2) return ERTM_EINVAL;
    const long long n = (long long)x->n * (x->h / 2) * (x->w / 2) * x->c;
    const long long rows = (long long)x->n * (x->h / 2);
    if (aligned16(y) && rows <= 65535) {
        const dim3 grid((x->w / 2 * (x->c / 8) + 255) / 256, (unsigned)rows);
        k_pool_fwd8<<<grid, 256, 0, (cudaStream_t)stream>>>(act_of(x), reinterpret_cast<uint4*>(y));
        return rc_of(cudaGetLastError());
    }
    k_pool_fwd<<<grid_of(n), 256, 0, (cudaStream_t)stream>>>(act_of(x), reinterpret_cast<bf16*>(y), n);
    return rc_of(cudaGetLastError());
}

int ertm_nn_pool2_bwd(const ertm_nn_act* x, const void* dy, const ertm_nn_act* dx, int relu_mask, void* stream)
{
    if (!act_ok(x) || !dy || !act_ok(dx) || x->h % 2 || x->w % 2) return ERTM_EINVAL;
    if (dx->cstride != x->cstride || dx->coff != x->coff || dx->c != x->c) return ERTM_EINVAL;
    const long long n = (long long)x->n * (x->h / 2) * (x->w / 2) * x->c;
    // the gradient lands at the same offsets as x's elements (same view layout)
    Act xa = act_of(x);
    bf16* dxp = reinterpret_cast<bf16*>(const_cast<void*>(dx->data));
    const long long rows = (long long)x->n * (x->h / 2);
    if (aligned16(dy) && rows <= 65535) {
        const dim3 grid((x->w / 2 * (x->c / 8) + 255) / 256, (unsigned)rows);
        k_pool_bwd8<<<grid, 256, 0, (cudaStream_t)stream>>>(xa, reinterpret_cast<const uint4*>(dy), dxp, relu_mask);
        return rc_of(cudaGetLastError());
    }
    k_pool_bwd<<<grid_of(n), 256, 0, (cudaStream_t)stream>>>(xa, reinterpret_cast<const bf16*>(dy), dxp, n,
                                                             relu_mask);
    return rc_of(cudaGetLastError());
}

int ertm_nn_bias_grad(const ertm_nn_act* dy, float* db, void* stream)
{
    if (!act_ok(dy) || !db) return ERTM_EINVAL;
    const long long P = (long long)dy->n * dy->h * dy->w;
    // about 64 pixels or more per thread, at most four blocks per SM
    const int cb = std::min(32, dy->c / 8);
    const dim3 grid((unsigned)std::max(1LL, std::min(P * cb / (256 * 16), 4LL * 148)), (dy->c / 8 + 31) / 32);
    k_bias_grad<<<grid, 256, 0, (cudaStream_t)stream>>>(act_of(dy), P, db);
    return rc_of(cudaGetLastError());
}

int ertm_nn_mse(const float* y, const float* target, int cstride, int c, long long pixels, float scale, void* grad,
                float* loss, void* stream)
{
    if (!y || !target || !grad || !loss || c > cstride || cstride % 8) return ERTM_EINVAL;
    k_mse<<<grid_of(pixels * (cstride / 8)), 256, 0, (cudaStream_t)stream>>>(
        y, target, cstride, c, pixels, scale, reinterpret_cast<bf16*>(grad), loss, aligned16(grad));
    return rc_of(cudaGetLastError());
}

int ertm_nn_adam(float* w, const float* g, float* m, float* v, void* wb, long long n, float lr, float b1, float b2,
                 float eps, int step, void* stream)
{
    if (!w || !g || !m || !v || !wb || n < 0 || step < 1) return ERTM_EINVAL;
    const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
    k_adam<<<grid_of(n), 256, 0, (cudaStream_t)stream>>>(w, g, m, v, reinterpret_cast<bf16*>(wb), n, lr, b1, b2, eps,
                                                         c1, c2);
    return rc_of(cudaGetLastError());
}

int ertm_nn_flip3(const void* w, void* wf, int co, int ci, void* stream)
{
    if (!w || !wf || co < 1 || ci < 1) return ERTM_EINVAL;
    k_flip3<<<grid_of((long long)co * 9 * ci), 256, 0, (cudaStream_t)stream>>>(reinterpret_cast<const bf16*>(w),
                                                                             reinterpret_cast<bf16*>(wf), co, ci);
    return rc_of(cudaGetLastError());
}

int ertm_nn_transpose(const void* a, void* t, int rows, int cols, void* stream)
{
    if (!a || !t || rows < 1 || cols < 1) return ERTM_EINVAL;
    k_transpose<<<grid_of((long long)rows * cols), 256, 0, (cudaStream_t)stream>>>(
        reinterpret_cast<const bf16*>(a), reinterpret_cast<bf16*>(t), rows, cols);
    return rc_of(cudaGetLastError());
}

int ertm_nn_to_bf16(const float* a, void* b, long long n, void* stream)
{
    if (!a || !b || n < 0) return ERTM_EINVAL;
    k_f32_to_bf16<<<grid_of(n), 256, 0, (cudaStream_t)stream>>>(a, reinterpret_cast<bf16*>(b), n);
    return rc_of(cudaGetLastError());
}

int ertm_nn_run(const ertm_nn_op* ops, int nops, void* const* ptr, int nptr, int* done, int* err, void* stream)
{
    if (done) *done = 0;
    if (nops < 0 || nptr < 0 || (nops && !ops) || (nptr && !ptr)) return ERTM_EINVAL;
    int i = 0, rc = ERTM_OK;
    while (i < nops && rc == ERTM_OK) {
        const ertm_nn_op& o = ops[i];
        void* p[3];
        for (int q = 0; q < 3; q++) {
            if (o.p[q] >= nptr) return ERTM_EINVAL;
            p[q] = o.p[q] < 0 ? nullptr : ptr[o.p[q]];
        }
        const ertm_nn_act* mask = o.flag ? &o.m : nullptr;
        int used = 1;
        switch (o.kind) {
        case ERTM_NN_OP_CONV:
            rc = ertm_nn_conv3x3(&o.a, p[0], (const float*)p[1], &o.b, o.flag, (float*)p[2], err, stream);
            break;
        case ERTM_NN_OP_CONV_DGRAD: rc = ertm_nn_conv3x3_dgrad(&o.a, p[0], &o.b, mask, err, stream); break;
        case ERTM_NN_OP_CONV_WGRAD:
            rc = ertm::nn_conv3x3_wgrad(&o.a, &o.b, (float*)p[0], (float*)p[1], ertm::kSplitsOfPlan, err, stream);
            break;
        case ERTM_NN_OP_UP: rc = ertm_nn_up2(&o.a, p[0], (const float*)p[1], &o.b, o.flag, err, stream); break;
        case ERTM_NN_OP_UP_DGRAD: rc = ertm_nn_up2_dgrad(&o.a, p[0], &o.b, mask, err, stream); break;
        case ERTM_NN_OP_UP_WGRAD:
            rc = ertm::nn_up2_wgrad(&o.a, &o.b, (float*)p[0], (float*)p[1], ertm::kSplitsOfPlan, err, stream);
            break;
        case ERTM_NN_OP_POOL: rc = ertm_nn_pool2(&o.a, p[0], stream); break;
        case ERTM_NN_OP_POOL_BWD: rc = ertm_nn_pool2_bwd(&o.a, p[0], &o.b, o.flag, stream); break;
        case ERTM_NN_OP_ZERO: {
            ertm::ZeroList z;
            for (used = 0; i + used < nops && used < ertm::ZERO_MAX && ops[i + used].kind == ERTM_NN_OP_ZERO; used++) {
                const ertm_nn_op& f = ops[i + used];
                if (f.n < 1 || f.p[0] < 0 || f.p[0] >= nptr || !ptr[f.p[0]]) return ERTM_EINVAL;
                z.add(ptr[f.p[0]], f.n);
            }
            rc = rc_of(ertm::launch_zero(z, (cudaStream_t)stream));
            break;
        }
        case ERTM_NN_OP_PACK: {
            if (!act_ok(&o.b) || o.b.cstride != 8 || o.b.c != 8 || !p[0] || o.flag < 1 || o.flag > 8) return ERTM_EINVAL;
            const long long n = (long long)o.b.n * o.b.h * o.b.w;
            k_pack8<<<grid_of(n), 256, 0, (cudaStream_t)stream>>>((const float*)p[0],
                                                                 (uint4*)const_cast<void*>(o.b.data), o.flag, n);
            rc = rc_of(cudaGetLastError());
            break;
        }
        default: return ERTM_EINVAL;
        }
        if (rc == ERTM_OK) i += used;
        if (done) *done = i;
    }
    return rc;
}

}  // extern "C"
