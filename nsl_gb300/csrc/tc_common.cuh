// Blackwell (sm_100 family) tensor-core plumbing in inline PTX: mbarriers, TMA tile loads, tcgen05 MMA / TMEM.
//
// Every wait on an mbarrier is bounded: after MBAR_SPIN_LIMIT polls the waiter records an error code in a global
// flag and gives up, so a kernel that loses a signal returns instead of hanging the GPU.
#pragma once

#include <cuda.h>
#include <stdint.h>

namespace nslg {
namespace tc {

constexpr uint32_t MBAR_SPIN_LIMIT = 1u << 24;  // try_wait polls (each may suspend briefly): seconds, not forever

__device__ __forceinline__ uint32_t smem_addr(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}

// One arrival (count 1) on a CTA-local mbarrier.
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t phase) {
    uint32_t ok;
    asm volatile(
        "{\n"
        " .reg .pred p;\n"
        " mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(phase)
        : "memory");
    return ok != 0;
}

// Bounded wait for the phase with parity `phase` to complete. Returns false (and sets *err) on timeout.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t phase, int *err, int code) {
    for (uint32_t i = 0; i < MBAR_SPIN_LIMIT; ++i)
        if (mbar_try_wait(bar, phase)) return true;
    if (err) atomicExch(err, code);
    return false;
}

// 2-D tiled TMA load into shared memory, completion signalled on `bar` (complete_tx bytes).
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int x, int y, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            smem_addr(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_addr(bar))
        : "memory");
}

// Contiguous bulk copy into shared memory (addresses and size multiples of 16 bytes), completion on `bar`.
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(dst)),
                 "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}

__device__ __forceinline__ void prefetch_tmap(const CUtensorMap *map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

// Make generic-proxy shared-memory writes visible to the async proxy (TMA, tensor core).
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// ----- TMEM ------------------------------------------------------------------------------------------------------
// Allocation by one full warp; the TMEM address is written to *dst (shared memory).
__device__ __forceinline__ void tmem_alloc(uint32_t *dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(dst)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// D[tmem] (+)= A[smem] * B[smem]^T, kind::tf32, cta_group::1, issued by one thread.
__device__ __forceinline__ void mma_tf32(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n"
        " .reg .pred p;\n"
        " setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// Arrive on `bar` once every tcgen05.mma issued so far by this thread has completed.
__device__ __forceinline__ void mma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                     smem_addr(bar))
                 : "memory");
}

// 32 lanes x 8 consecutive 32-bit columns; the warp reads its own 32-lane quarter of TMEM. (The register fences keep the
// compiler from using a result before the wait, which does not name the registers.)
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8]) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        asm volatile("" : "+r"(r[i]));
        v[i] = __uint_as_float(r[i]);
    }
}

// 32 lanes x 8 columns without waiting: several loads may be in flight; call tmem_wait_ld before reading r.
__device__ __forceinline__ void tmem_ld8_async(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
}

// Waits for this thread's outstanding tcgen05.ld; the register fence keeps the compiler from reading r earlier.
template <int N>
__device__ __forceinline__ void tmem_wait_ld(uint32_t (&r)[N][8]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int a = 0; a < N; ++a)
#pragma unroll
        for (int i = 0; i < 8; ++i) asm volatile("" : "+r"(r[a][i]));
}

// Shared-memory matrix descriptor: K-major operand, 128-byte swizzle, 8-row core groups 1024 B apart.
__device__ __forceinline__ uint64_t sdesc_kmajor_sw128(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFF);  // start address
    d |= (uint64_t)1 << 16;                  // leading byte offset (unused for swizzled K-major)
    d |= (uint64_t)(1024 >> 4) << 32;        // stride byte offset: next 8-row group
    d |= (uint64_t)1 << 46;                  // descriptor version (sm_100)
    d |= (uint64_t)2 << 61;                  // layout: SWIZZLE_128B
    return d;
}

// Shared-memory matrix descriptor: K-major operand rows of 32 B, 32-byte swizzle, 8-row core groups 256 B apart.
__device__ __forceinline__ uint64_t sdesc_kmajor_sw32(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFF);
    d |= (uint64_t)1 << 16;           // leading byte offset (unused for swizzled K-major)
    d |= (uint64_t)(256 >> 4) << 32;  // stride byte offset: 8 rows x 32 B
    d |= (uint64_t)1 << 46;           // descriptor version (sm_100)
    d |= (uint64_t)6 << 61;           // layout: SWIZZLE_32B
    return d;
}

__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
    return (1u << 4)     // D: F32
           | (1u << 7)   // A: BF16
           | (1u << 10)  // B: BF16
           | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// D[tmem] (+)= A[smem] * B[smem]^T, kind::f16 (BF16 operands, FP32 accumulation), issued by one thread.
// (The A collector buffer does not change the instruction rate measured on this part, ~44 cycles per N = 32 MMA.)
__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(
            d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// Instruction descriptor, kind::tf32 with FP32 accumulation, both operands K-major.
__host__ __device__ constexpr uint32_t idesc_tf32(int M, int N) {
    return (1u << 4)                      // D format: F32
           | (2u << 7)                    // A format: TF32
           | (2u << 10)                   // B format: TF32
           | ((uint32_t)(N >> 3) << 17)   // N / 8
           | ((uint32_t)(M >> 4) << 24);  // M / 16
}

// Byte offset of element (row, k) (4-byte elements) in a K-major 128B-swizzled tile of 32-element rows.
__device__ __forceinline__ uint32_t sw128_offset(int row, int k) {
    const int chunk = (k >> 2) ^ (row & 7);
    return (uint32_t)(row * 128 + chunk * 16 + (k & 3) * 4);
}

// Split of a double into tf32 hi (low 13 mantissa bits of the float cleared) and an fp32 remainder.
__device__ __forceinline__ void split_tf32(double v, float &hi, float &lo) {
    const float f = (float)v;
    hi = __uint_as_float(__float_as_uint(f) & 0xFFFFE000u);
    lo = (float)(v - (double)hi);
}

// The same split without FP64 arithmetic (conversions and subtractions of FP64 numbers run on the FP64 pipe, ~2 per clock per
// SM): f = v rounded to FP32 from the bit pattern, hi = f with 13 bits cleared, lo = (f - hi) + (v - f), the second term an
// integer of 30 bits at a power-of-two scale. hi is the same bit for bit, lo to its last bit (the tensor core reads lo's
// upper 11).
__device__ __forceinline__ void split_tf32_int(double v, float &hi, float &lo) {
    const unsigned h32 = (unsigned)__double2hiint(v), l32 = (unsigned)__double2loint(v);
    const int e = (int)(h32 >> 20 & 0x7FFu) - 896;  // FP32's biased exponent
    if (((h32 << 1) | l32) == 0u) {  // zero (padding)
        hi = lo = 0.f;
        return;
    }
    if (e < 53 || e > 253) {  // hi or lo outside the normal range of FP32, infinities, NaN
        split_tf32(v, hi, lo);
        return;
    }
    unsigned fb = __funnelshift_l(l32, h32 & 0x7FFFFFFFu, 3) - (896u << 23);  // truncated to 24 bits
    int g = (int)(l32 & 0x1FFFFFFFu);                                          // what was cut off, units of ulp 2^-29
    if (g > 0x10000000 || (g == 0x10000000 && (fb & 1u))) {                    // round to nearest even
        ++fb;
        g -= 0x20000000;
    }
    const unsigned hb = fb & 0xFFFFE000u, sign = h32 & 0x80000000u;
    const float l = fmaf((float)g, __uint_as_float((unsigned)(e - 52) << 23),
                         __uint_as_float(fb) - __uint_as_float(hb));
    hi = __uint_as_float(hb | sign);
    lo = __uint_as_float(__float_as_uint(l) ^ sign);
}

// (double)v in integer arithmetic for normal v.
__device__ __forceinline__ double widen_int(float v) {
    const unsigned u = __float_as_uint(v), e = u >> 23 & 0xFFu;
    if (e == 0u || e == 255u) return (double)v;
    return __longlong_as_double((long long)(((unsigned long long)(u & 0x80000000u) << 32) |
                                            (((unsigned long long)(u & 0x7FFFFFFFu) + (896ull << 23)) << 29)));
}

}  // namespace tc
}  // namespace nslg
