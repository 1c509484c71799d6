// gb_tc05.h -- inline-PTX primitives for the 5th-generation tensor cores
// (tcgen05: TMEM accumulators, shared-memory operand descriptors, mbarriers)
// and the error-free FP64 digit splitting shared by the tensor-core kernels.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

// ---------------------------------------------------------------- addresses, fences
__device__ __forceinline__ uint32_t tc_smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void tc_fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ uint64_t tc_globaltimer()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// ---------------------------------------------------------------- TMEM
// allocation by one whole warp; the TMEM address is written to smem[dst]
__device__ __forceinline__ void tc_tmem_alloc(uint32_t dst_smem, uint32_t ncols)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_tmem_dealloc(uint32_t taddr, uint32_t ncols)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

__device__ __forceinline__ void tc_tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// ---------------------------------------------------------------- mbarrier
__device__ __forceinline__ void tc_mbar_init(uint32_t bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ bool tc_mbar_try_wait(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(bar), "r"(parity)
                 : "memory");
    return ok != 0;
}
__device__ __forceinline__ void tc_mbar_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// arrival that also expects `bytes` of asynchronous copies to complete on the barrier
__device__ __forceinline__ void tc_mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// bulk copy global -> shared (16-byte aligned addresses, size a multiple of 16),
// completing its bytes on the mbarrier
__device__ __forceinline__ void tc_bulk_g2s(uint32_t dst_smem, const void *src, uint32_t bytes, uint32_t bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     dst_smem),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
// asynchronous copies of the issuing thread: global -> shared, zero filled past src_bytes
__device__ __forceinline__ void tc_cp8(uint32_t dst_smem, const void *src, uint32_t src_bytes)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst_smem), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void tc_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// until at most PENDING of this thread's groups are in flight
template <int PENDING>
__device__ __forceinline__ void tc_cp_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
}
// bounded wait for the phase of the given parity; false after limit_ns
__device__ __forceinline__ bool tc_mbar_wait(uint32_t bar, uint32_t parity, uint64_t limit_ns)
{
    if (tc_mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = tc_globaltimer();
    while (!tc_mbar_try_wait(bar, parity))
        if (tc_globaltimer() - t0 > limit_ns) return false;
    return true;
}

// ---------------------------------------------------------------- MMA
// shared-memory matrix descriptor, no swizzle: 8-row x 16-byte core matrices of
// 128 contiguous bytes; lbo = byte distance of core matrices adjacent in K,
// sbo = byte distance of core matrices adjacent in M (or N)
__device__ __forceinline__ uint64_t tc_sdesc(uint32_t saddr, uint32_t lbo, uint32_t sbo)
{
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) |
           (1ull << 46);
}
// instruction descriptor of kind::f16: f16 x f16 -> f32, both K-major, M x N
__host__ __device__ constexpr uint32_t tc_idesc_f16(int M, int N)
{
    return (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
// D[tmem] (+)= A[smem] * B[smem]^T (kind::f16, types from idesc), issued by one thread
__device__ __forceinline__ void tc_mma_kf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                            uint32_t accumulate)
{
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "setp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
                 "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
                 : "memory");
}
// mbarrier arrive once all tcgen05 operations issued so far by this thread are done
__device__ __forceinline__ void tc_mma_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}

// ---------------------------------------------------------------- error-free digit splitting
// An FP64 entry x of a row (or column) with scale 2^e (|x| < 2^e over the row)
// is the integer T = x 2^(53 - e) rounded to nearest, |T| <= 2^53, i.e. exact to
// half a unit of 2^(e - 53). With the bias B = 0x80808080808080, U = T + B lies
// in [0, 2^56) and its seven bytes b_0 (least significant) .. b_6 give balanced
// digits d_p = b_(6-p) - 128:
//   x = sum_p d_p 2^(-8p) 2^(e - 5),   p = 0 (most significant) .. 6,
// with d_0 in [-32, 32] and d_1 .. d_6 in [-128, 127]. Only integer operations
// touch x; every digit is exact in f16 (and bf16).
//
// Exact accumulation bound: the digit products of level L = p + q are at most
// 2^12 for the two pairs with p = 0 or q = 0 and 2^14 for the others, so a
// level sums to at most 2^13 + 5 * 2^14 per term (L = 6) and stays below 2^24
// -- an exact FP32 integer -- for up to OZ_EXACT_TERMS terms.
#define OZ_DIGITS 7
#define OZ_NO_EXP (-2000)          // scale of an all-zero row or column
#define OZ_EXACT_TERMS 186
#define OZ_SCALE_OFFSET 10         // a digit product of level 0 carries 2^(e + f - 10)

// exponent contribution of one entry: |x| < 2^(ex - 1022); OZ_NO_EXP for 0 and subnormals
__device__ __forceinline__ int oz_exponent(double x)
{
    const int ex = (int)((__double_as_longlong(x) >> 52) & 0x7ff);
    return ex ? ex - 1022 : OZ_NO_EXP;
}
#include "gb_ozconv.h"
// U 2^8 of one entry, sb = its scale + OZ_SHIFT0 (OZ_SHIFT_NONE: no digits)
__device__ __forceinline__ unsigned long long oz_bias(double x, int sb)
{
    return oz_digits((uint32_t)__double2hiint(x), (uint32_t)__double2loint(x), sb);
}
// the seven digits of two entries (oz_digits) as f16x2 words, u0's in the low half, most
// significant first: byte b goes under 0x64 as 0x64bb = 1024 + b, from which 1152 is
// subtracted, both exact. A byte permute pairs two bytes of both entries, a second one
// spreads each pair over the constant: 11 for seven digits.
__device__ __forceinline__ void oz_pack(unsigned long long u0, unsigned long long u1, uint32_t d[OZ_DIGITS])
{
    const uint32_t l0 = (uint32_t)u0, h0 = (uint32_t)(u0 >> 32), l1 = (uint32_t)u1, h1 = (uint32_t)(u1 >> 32);
    const uint32_t ha = __byte_perm(h0, h1, 0x7362), hb = __byte_perm(h0, h1, 0x5140);
    const uint32_t la = __byte_perm(l0, l1, 0x7373), lb = __byte_perm(l0, l1, 0x6251);
    d[0] = __byte_perm(ha, 0x64646464u, 0x4342);
    d[1] = __byte_perm(ha, 0x64646464u, 0x4140);
    d[2] = __byte_perm(hb, 0x64646464u, 0x4342);
    d[3] = __byte_perm(hb, 0x64646464u, 0x4140);
    d[4] = __byte_perm(la, 0x64646464u, 0x4140);
    d[5] = __byte_perm(lb, 0x64646464u, 0x4342);
    d[6] = __byte_perm(lb, 0x64646464u, 0x4140);
#pragma unroll
    for (int p = 0; p < OZ_DIGITS; ++p) asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(d[p]) : "r"(d[p]), "r"(0x64806480u));
}

// levels (exact FP32 integers) -> hi (levels 0-2, units 2^-16) and lo (levels 3-7,
// units 2^-56) of one output
__device__ __forceinline__ void oz_levels_to_int(const float *v, long long &hi, long long &lo)
{
    hi = ((long long)__float2int_rn(v[1]) * 256 + __float2int_rn(v[2])) + (long long)__float2int_rn(v[0]) * 65536;
    lo = (((long long)__float2int_rn(v[6]) * 256 + __float2int_rn(v[7])) + (long long)__float2int_rn(v[5]) * 65536) +
         (long long)__float2int_rn(v[4]) * 16777216 + ((long long)__float2int_rn(v[3]) << 32);
}
