// gb_coop.h -- barrier words of a cooperative grid: arrivals counted in one word,
// release by a second one that carries a generation and a 32-bit message, so that
// a waiting block learns both in one trip to L2. Waits are bounded by the callers
// (COOP_WAIT_NS of %globaltimer; the longest phase of a kernel is below a second). A
// launch stalled on purpose (GCGE_GPU_TestStallGridWait) finds the count of arrivals off,
// so that its first barrier never completes, and waits COOP_STALL_NS. (The barriers
// themselves are the same: a test of a flag or of an argument before the arrival took 20
// to 60 ns of a barrier's 2.2 us.)
#pragma once
#include <cuda_runtime.h>

#include "gb_internal.h"

#define COOP_WAIT_NS 20000000000ull
#define COOP_STALL_NS 100000000ull

__device__ __forceinline__ unsigned long long coop_now()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ unsigned coop_arrive(unsigned *w)
{
    unsigned t;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(t) : "l"(w) : "memory");
    return t;
}
__device__ __forceinline__ unsigned long long coop_ld64(const unsigned *w)
{
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(w) : "memory");
    return v;
}
__device__ __forceinline__ unsigned coop_ld32(const unsigned *w)
{
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(w) : "memory");
    return v;
}
// the limit of the next launch's waits; a stall is for one launch
static inline unsigned long long gb_coop_wait_ns(gcge_gpu_ctx *ctx)
{
    if (!ctx->coop_stall) return COOP_WAIT_NS;
    ctx->coop_stall = 0;
    cudaMemsetAsync(ctx->dev_bar, 0x40, sizeof(unsigned), ctx->stream);
    return COOP_STALL_NS;
}
// word pair w (8-byte aligned): generation gen, message msg
__device__ __forceinline__ void coop_release(unsigned *w, unsigned gen, unsigned msg)
{
    asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(w), "l"((unsigned long long)gen << 32 | msg) : "memory");
}
