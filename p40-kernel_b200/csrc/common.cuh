// common.cuh -- device helpers shared by every kernel of the sm_100a build.
//
// Arithmetic rules (they make the device output equal the reference's HOST code bit for bit):
//   * every fp32 operation that the host performs is issued as one explicit IEEE operation
//     (__fmul_rn / __fadd_rn / __fdiv_rn), so the compiler can neither fuse nor approximate it;
//   * fp32 -> fp16 uses the host's ties-away rule, not the hardware ties-to-even conversion;
//   * float -> int uses ties-away (lroundf semantics), not ties-to-even.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200 {

constexpr int W_BLOCK_BYTES = 34;   // PQ2_0 block: fp16 scale + 32 code bytes (128 weights)
constexpr int A_BLOCK_BYTES = 36;   // Q8_1 block: fp16 scale + int16 sum + 32 int8
constexpr int FWHT_N = 1024;

// Sticky status word: bounded waits write a non-zero code here instead of spinning forever.
__device__ int g_device_status = 0;

enum : int { STATUS_OK = 0, STATUS_MBARRIER_TIMEOUT = 1, STATUS_GRID_TIMEOUT = 2 };

// ---- fp16 <-> fp32 -------------------------------------------------------------------------
__device__ __forceinline__ float f16_bits_to_f32(uint32_t h) {
    return __half2float(__ushort_as_half((unsigned short)h));   // exact widening
}

// Host rule of the reference (src/p40_common.h:91-112): the first dropped mantissa bit alone
// decides the bump, i.e. nearest with ties away from zero; subnormals and overflow included.
__device__ __forceinline__ uint32_t f32_to_f16_bits_ties_away(float f) {
    const uint32_t x = __float_as_uint(f);
    const uint32_t sign = (x >> 16) & 0x8000u;
    const uint32_t e8 = (x >> 23) & 255u;
    const uint32_t frac = x & 0x7FFFFFu;
    if (e8 == 255u) return sign | 0x7C00u | (frac ? 0x200u : 0u);
    int e = (int)e8 - 112;
    if (e >= 31) return sign | 0x7C00u;
    if (e <= 0) {
        if (e < -10) return sign;
        const uint32_t full = frac | 0x800000u;
        const uint32_t sh = (uint32_t)(14 - e);
        return sign | ((full >> sh) + ((full >> (sh - 1)) & 1u));
    }
    uint32_t q = (frac >> 13) + ((frac >> 12) & 1u);
    if (q == 1024u) { q = 0; e += 1; if (e >= 31) return sign | 0x7C00u; }
    return sign | ((uint32_t)e << 10) | q;
}

// lroundf semantics for |t| < 2^23 (a NaN gives 0, as the host's conversion does on x86-64): towards zero behind the largest float below a half, which takes
// every t whose fraction is a half or more across the next integer and no other (all 2.5 x 10^9 floats of that range, of either sign, were compared).
__device__ __forceinline__ int round_ties_away(float t) { return __float2int_rz(__fadd_rn(t, copysignf(0x1.fffffep-2f, t))); }

// The same, five instructions longer.  For the list launch, whose multiply comes out of the compiler differently with every change around it: with the short
// form in its quantiser the layer sweep, which quantises nothing, takes 118.9 us instead of 115.3 (the decode step 3152 instead of 3163).
__device__ __forceinline__ int round_ties_away_long(float t) {
    const float r = truncf(t);
    const float frac = __fsub_rn(t, r);          // exact
    int q = (t == t) ? (int)r : 0;
    if (fabsf(frac) >= 0.5f) q += (t < 0.0f) ? -1 : 1;
    return q;
}

// ---- two fp32 operations in one instruction, each rounded as __fmaf_rn and __fadd_rn ----
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("{\n\t"
        ".reg .b64 a, b, c, d;\n\t"
        "mov.b64 a, {%2, %3};\n\t"
        "mov.b64 b, {%4, %5};\n\t"
        "mov.b64 c, {%6, %7};\n\t"
        "fma.rn.f32x2 d, a, b, c;\n\t"
        "mov.b64 {%0, %1}, d;\n\t"
        "}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    float2 d;
    asm("{\n\t"
        ".reg .b64 a, b, d;\n\t"
        "mov.b64 a, {%2, %3};\n\t"
        "mov.b64 b, {%4, %5};\n\t"
        "add.rn.f32x2 d, a, b;\n\t"
        "mov.b64 {%0, %1}, d;\n\t"
        "}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}

// ---- integer dot ------------------------------------------------------------------------------
// Four unsigned bytes of `w` times four signed bytes of `a`, plus c (reference: the host dp4a
// emulation, src/p40_common.h:131-140, applied to codes 0..3 which are non-negative either way).
__device__ __forceinline__ int dp4a_us(uint32_t w, int a, int c) {
    int r;
    asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(r) : "r"(w), "r"(a), "r"(c));
    return r;
}

// Sum over one 32-weight chunk of code * activation.  w0 / w1 are the two 16-code words, a[0..7] the
// eight activation words of the permuted Q8_1 block: field k of word w pairs with activation word
// 4w + k (src/pq2_0.h:155-166).  Fields are masked in place, so the four field sums come out scaled
// by 64, 16, 4 and 1; they are four independent dp4a chains (the scheduler can overlap them), joined
// as (s3 + 4 s2 + 16 s1 + 64 s0) >> 6, which is exact because the sum is a multiple of 64.  Callers
// pass init64 = -64 * s so that the result is (sum code*a) - s.
__device__ __forceinline__ int chunk_sumi_scaled(uint32_t w0, uint32_t w1, const int (&a)[8], int init64) {
    int s3 = dp4a_us(w0 & 0xC0C0C0C0u, a[3], init64);
    int s2 = dp4a_us(w0 & 0x30303030u, a[2], 0);
    int s1 = dp4a_us(w0 & 0x0C0C0C0Cu, a[1], 0);
    int s0 = dp4a_us(w0 & 0x03030303u, a[0], 0);
    s3 = dp4a_us(w1 & 0xC0C0C0C0u, a[7], s3);
    s2 = dp4a_us(w1 & 0x30303030u, a[6], s2);
    s1 = dp4a_us(w1 & 0x0C0C0C0Cu, a[5], s1);
    s0 = dp4a_us(w1 & 0x03030303u, a[4], s0);
    return (s3 + (s2 << 2) + (s1 << 4) + (s0 << 6)) >> 6;
}

// ---- shared-memory barriers and bulk copies (sm_90+ PTX, every copy is local to its CTA) -------
__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Adds 1 to a counter in global memory; what the CTA wrote before the barrier in front of this call is visible to whoever
// reads the sum, and what they wrote to this CTA after the barrier behind it.
__device__ __forceinline__ unsigned int count_arrival(unsigned int *counter) {
    unsigned int old;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(old) : "l"(counter) : "memory");
    return old;
}
// ---- clusters of CTAs ----
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Into CTA `rank`'s shared memory, at the place that p is in this one's (aligned to what is stored), counted on its barrier at the place of `bar`.
__device__ __forceinline__ void st_async_u32(const void *p, uint64_t *bar, uint32_t rank, uint32_t a) {
    asm volatile("{\n\t.reg .u32 x, y;\n\tmapa.shared::cluster.u32 x, %0, %2;\n\tmapa.shared::cluster.u32 y, %1, %2;\n\t"
                 "st.async.shared::cluster.mbarrier::complete_tx::bytes.u32 [x], %3, [y];\n\t}"
                 ::"r"(smem_u32(p)), "r"(smem_u32(bar)), "r"(rank), "r"(a) : "memory");
}
__device__ __forceinline__ void st_async_f32x2(const float *p, uint64_t *bar, uint32_t rank, float a, float b) {
    asm volatile("{\n\t.reg .u32 x, y;\n\tmapa.shared::cluster.u32 x, %0, %2;\n\tmapa.shared::cluster.u32 y, %1, %2;\n\t"
                 "st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [x], {%3, %4}, [y];\n\t}"
                 ::"r"(smem_u32(p)), "r"(smem_u32(bar)), "r"(rank), "f"(a), "f"(b) : "memory");
}
__device__ __forceinline__ void st_async_f32x4(const float *p, uint64_t *bar, uint32_t rank, float a, float b, float c, float d) {
    asm volatile("{\n\t.reg .u32 x, y;\n\tmapa.shared::cluster.u32 x, %0, %2;\n\tmapa.shared::cluster.u32 y, %1, %2;\n\t"
                 "st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [x], {%3, %4, %5, %6}, [y];\n\t}"
                 ::"r"(smem_u32(p)), "r"(smem_u32(bar)), "r"(rank), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
// Bounded wait: returns false (and records the status word) instead of spinning forever.  The
// barrier is polled with the non-blocking test; between polls the thread sleeps first_ns, 2 first_ns, ... max_ns,
// which keeps a waiting warp off the issue ports (the blocking form of the wait expands to a
// software time-out loop of a couple of dozen instructions per poll).
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity, uint32_t first_ns = 32,
                                                  uint32_t max_ns = 256) {
    uint32_t ok;
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        ".reg .u32 n, ns;\n\t"
        "mov.u32 n, %3;\n\t"
        "mov.u32 ns, %4;\n\t"
        "mov.u32 %0, 1;\n\t"
        "WAIT_LOOP:\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "@p bra WAIT_DONE;\n\t"
        "nanosleep.u32 ns;\n\t"
        "add.u32 ns, ns, ns;\n\t"
        "min.u32 ns, ns, %5;\n\t"
        "sub.u32 n, n, 1;\n\t"
        "setp.ne.u32 p, n, 0;\n\t"
        "@p bra WAIT_LOOP;\n\t"
        "mov.u32 %0, 0;\n\t"
        "WAIT_DONE:\n\t"
        "}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity), "r"(1u << 22), "r"(first_ns), "r"(max_ns)
        : "memory");
    if (!ok) atomicExch(&g_device_status, STATUS_MBARRIER_TIMEOUT);
    return ok != 0;
}
// The same wait for a barrier that is expected within a fraction of a microsecond (a tensor-core result, a stage a
// neighbouring role is about to hand over): polls back to back first, and sleeps between polls only when that did
// not help.  Bounded like the one above.
__device__ __forceinline__ bool mbar_wait_hot(uint64_t *bar, uint32_t parity) {
    uint32_t ok = 0;
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        ".reg .u32 n;\n\t"
        "mov.u32 n, 512;\n\t"
        "mov.u32 %0, 1;\n\t"
        "HOT_LOOP:\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "@p bra HOT_DONE;\n\t"
        "sub.u32 n, n, 1;\n\t"
        "setp.ne.u32 p, n, 0;\n\t"
        "@p bra HOT_LOOP;\n\t"
        "mov.u32 %0, 0;\n\t"
        "HOT_DONE:\n\t"
        "}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
    return mbar_wait_bounded(bar, parity, 32, 128);
}
__device__ __forceinline__ unsigned long long global_timer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ uint32_t global_timer_ms() { return (uint32_t)(global_timer_ns() >> 20); }       // steps of 1.05 ms
// The blocking form of the test: the unit gives the thread back when the phase has completed, after suspend_ns at the latest.
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity, uint32_t suspend_ns) {
    uint32_t ok;
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity), "r"(suspend_ns)
        : "memory");
    return ok != 0;
}
// The bounded wait in the blocking form: a dozen warps that wait for the same thing need no sleeps between their polls.  Between two
// suspensions a thread looks at *stop and at the clock.  False when *stop was set -- by a thread of the CTA that has given up, and said
// so, on something that this one waits for in the end -- or when limit_ms milliseconds have passed (status word; *stop is set).
constexpr uint32_t MBAR_SUSPEND_NS = 10000;
__device__ __forceinline__ bool mbar_wait_suspended(uint64_t *bar, uint32_t parity, volatile int *stop, uint32_t limit_ms) {
    if (mbar_try_wait(bar, parity, MBAR_SUSPEND_NS)) return true;
    const uint32_t t0 = global_timer_ms();
    while (!mbar_try_wait(bar, parity, MBAR_SUSPEND_NS)) {
        if (*stop) return false;
        if (global_timer_ms() - t0 > limit_ms) {
            *stop = 1;
            atomicExch(&g_device_status, STATUS_MBARRIER_TIMEOUT);
            return false;
        }
    }
    return true;
}
// One non-blocking poll: has the phase with this parity completed?
__device__ __forceinline__ bool mbar_test(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// 1-D bulk copy global -> shared of `bytes` (multiple of 16, both addresses 16-byte aligned),
// completion counted on `bar`.
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar, uint64_t policy) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;"
        ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)), "l"(policy)
        : "memory");
}
// Asks L2 for `bytes` (multiple of 16, address 16-byte aligned).
__device__ __forceinline__ void bulk_prefetch_l2(const void *src, uint32_t bytes) {
    if (bytes) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}
// Asks L2 for the line at p.
__device__ __forceinline__ void prefetch_l2(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p) : "memory"); }
__device__ __forceinline__ uint64_t policy_evict_first() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ uint64_t policy_evict_normal() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(p));
    return p;
}
// Cache policy for data that many CTAs re-read (activation blocks of a token tile): keep it in L2.
__device__ __forceinline__ uint64_t policy_evict_last_or_default() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
    return p;
}
// Programmatic dependent launch: both are no-ops unless the launches carry the attribute.  Kernels call the wait first:
// a launch that starts early then has its direct predecessor to wait for and nothing older, which is why a mat-vec behind
// this library's quantiser may copy weights before its own wait.  What an earlier launch may have written is read through
// pointers without __restrict__ and with plain loads: a non-coherent one (ld.global.nc, __ldg) is for memory that nothing writes
// while the kernel is there, and may be moved in front of the wait.  (Weights of a mat-vec: plain loads too, unless only an
// option of the caller, who promises that nobody writes them, makes the kernel start early.)
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait_prior_grid() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// A kernel that never lets the next launch in lets it in by ending, CTA by CTA.  That is better where the kernel fills much of the chip and the next one has nothing to do
// before its own wait: its CTAs would go to what the running kernel leaves free, many on one SM and none on another, and stay there, or take issue slots and memory from
// it.  us, let in at the first instruction (or launched plainly) / at the end: 512 rows of 5120 RMSNorm + rotation with quantiser 14.4 / 11.5, of 3072 13.1 / 8.2, 148 of
// 5120 10.1 / 5.5, 700 of 1024 8.27 / 5.72; 37 x 17408 SwiGLU + the same 8.28 / 5.58, with the mat-mul 64 x 17408 44.8 / 41.1.  Few CTAs leave it room, and where the next kernel asks
// for its weights or its state first, early it is: one row's RMSNorm and SwiGLU in front of its projection (bonsai_p40_rmsnorm, bonsai_b200_swiglu), mat-vec behind its
// quantiser, list of delta-net steps, K/V calls (append 37.8 / 44.4, 5120 -> 64 3.16 / 3.56).

// A coherent load that stays behind the wait (both are volatile), and that the compiler may take in front of stores to shared memory.
__device__ __forceinline__ uint32_t ldg_u32(const void *p) {
    uint32_t v;
    asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ uint32_t ldg_nc_u16(const void *p) {
    unsigned short v;
    asm volatile("ld.global.nc.u16 %0, [%1];" : "=h"(v) : "l"(p));
    return v;
}

}  // namespace b200
