// tcgen05 building blocks shared by the tensor-core kernels (nn.cu, nn_conv.cu): bounded
// mbarrier waits, shared-memory and instruction descriptors, MMA issue, TMEM loads, and
// the NHWC activation view.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "ertm.h"
#include "ertm_internal.cuh"

namespace {

typedef __nv_bfloat16 bf16;

constexpr int BM = 128;      // rows per CTA (tcgen05 M)
constexpr unsigned kPolls = 1u << 24;

enum NnError { NN_OK = 0, NN_WAIT = 1 };

__device__ __forceinline__ uint32_t su32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* b, unsigned n)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(su32(b)), "r"(n) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t* b, unsigned parity)
{
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                 " selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(ok)
                 : "r"(su32(b)), "r"(parity)
                 : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_wait(uint64_t* b, unsigned parity)
{
    for (unsigned n = 0; n < kPolls; n++)
        if (mbar_try(b, parity)) return true;
    return false;
}

// shared-memory matrix descriptor, no swizzle: LBO = lbo bytes (to the core matrix next
// in K), SBO = sbo bytes (next in M or N)
__device__ __forceinline__ uint64_t sdesc(uint32_t saddr, uint32_t lbo, uint32_t sbo = 128)
{
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFF);
    d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
    d |= (uint64_t)1 << 46;   // descriptor version for sm_100
    return d;                  // base offset 0, legacy LBO mode, layout SWIZZLE_NONE
}

// instruction descriptor of kind::f16: BF16 x BF16 -> F32, both K-major, M = 128, N = n
__host__ __device__ constexpr uint32_t idesc_bf16(int n)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
}

__device__ __forceinline__ void umma(uint32_t tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc)
{
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n}\n" ::"r"(tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(acc), "r"(0), "r"(0), "r"(0), "r"(0)
        : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(su32(bar))
                 : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float* v)
{
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                   "=r"(r[7])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int q = 0; q < 8; q++) v[q] = __uint_as_float(r[q]);
}


// NHWC activation view: pixel p = (n*H + y)*W + x, channels [off, off+C) of a
// pixel stride of cs channels
struct Act {
    const bf16* p;
    int nb, h, w, cs, off, c;
};

inline int rc_of(cudaError_t e) { return e == cudaSuccess ? ERTM_OK : ERTM_ECUDA; }

inline Act act_of(const ertm_nn_act* a)
{
    return Act{reinterpret_cast<const bf16*>(a->data), a->n, a->h, a->w, a->cstride, a->coff, a->c};
}

// the operand copies move 16-byte chunks: every matrix starts on a 16-byte boundary
inline bool aligned16(const void* p) { return p && ((uintptr_t)p % 16) == 0; }
inline bool same_grid(const ertm_nn_act* a, const ertm_nn_act* b) { return a->n == b->n && a->h == b->h && a->w == b->w; }
inline bool act_ok(const ertm_nn_act* a)
{
    return a && a->data && a->n > 0 && a->h > 0 && a->w > 0 && a->c > 0 && a->c % 8 == 0 && a->coff % 8 == 0 &&
           a->cstride % 8 == 0 && a->coff + a->c <= a->cstride && ((uintptr_t)a->data % 16) == 0;
}
// a ReLU mask is read at the output's own element offsets
inline bool mask_ok(const ertm_nn_act* mask, const ertm_nn_act* dx)
{
    return !mask || (act_ok(mask) && same_grid(mask, dx) && mask->cstride == dx->cstride && mask->coff == dx->coff &&
                     mask->c == dx->c);
}

// 8 BF16 values of a 16-byte chunk
__device__ __forceinline__ void unpack8(const uint4& u, float* f)
{
    const uint32_t* w = &u.x;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        f[2 * q] = __uint_as_float(w[q] << 16);
        f[2 * q + 1] = __uint_as_float(w[q] & 0xffff0000u);
    }
}

}  // namespace

namespace ertm {
// ertm_nn_conv3x3_wgrad and ertm_nn_up2_wgrad with the bias gradient of the same dy, db += its
// sum over the pixels, in the same kernel (db NULL: none).
constexpr int kSplitsOfPlan = 1 << 30;   // splitk: as many as the plan takes
int nn_conv3x3_wgrad(const ertm_nn_act* x, const ertm_nn_act* dy, float* dw, float* db, int splitk, int* err,
                     void* stream);
int nn_up2_wgrad(const ertm_nn_act* x, const ertm_nn_act* dy, float* du, float* db, int splitk, int* err, void* stream);
}  // namespace ertm
