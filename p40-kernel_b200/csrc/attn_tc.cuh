// attn_tc.cuh -- causal attention of a prompt on the tensor cores (tcgen05.mma.kind::f16), fp32 in and out.
//
// attn_kernel (ops.cuh) multiplies on the CUDA cores and is bound by their issue slots and by shared memory.  Here both
// products run on the tensor cores without giving up fp32: every operand is scaled by a power of two (q and k per row, v per
// output dim and tile, softmax weights by 2^14) and split into two fp16 planes, high and low, 22 - 24 bits together; what
// the low plane cannot hold is below 2^-39 of the largest value under the same power of two.  The tensor core cuts the last bits of a sum off
// instead of rounding it, so sums are kept short: a score is six sums over 32 or 48 dims (an accumulator over all 256 was 1.5
// to 3 times less exact than the CUDA cores), joined by rounded additions, and a tile's weights x v go to a fresh accumulator
// that the CUDA cores add to the fp32 output.  Error against 64 bits: at
// ATC_MIN_TOKENS.
//
// attn_planes_kernel writes k and v once per call as tile images: the bytes that the attention kernel's shared memory holds
// for 64 keys of a kv head, planes split, swizzled and (v) transposed, fetched by one bulk copy each.  (Every CTA splitting
// its own tiles did that 50 times over at 2048 tokens and took twice the time of the products: 370 us.)
//
// attn_tc_kernel: CTA = 128 queries of one head, 512 threads, each one row and a quarter of its columns:
//   q . k, dims 0 .. 63      | outputs of the tile before into registers
//   q . k, dims 64 .. 255    |
//   (tensor core idle)       | softmax, weights -> planes in tensor memory
//   weights x v              |
// Shared memory: q high, k and v images of one tile, 64 KB each (K-major, 128-byte swizzle).  Tensor memory, all 512
// columns: 256 output (before that, sums of the scores), 128 scores (then weights), 128 q low.
// What bounds it (counted while a score was four sums): per tile 5900 of 10200 cycles were the tensor core's, most of them the score
// products (N = 64: it waits for the q rows from shared memory), the rest softmax and the exchanges in front of it.  us, CUDA cores / here, 24 heads over 4:
// 2048 tokens 2054 / 236, 1000 511 / 78, 600 196 / 52.
//
// A plane pair holds 2^-39 of the largest value under its power of two, so what is far smaller loses bits to values that a row may not
// even see.  A CTA whose queries and keys range too widely (atc_too_wide) does its queries again on the CUDA cores (attn_simt), with
// that kernel's results; so does one that meets an infinity, NaN or a value past 2^60.
#pragma once

#include "gemm_tc16.cuh"
#include "kv.cuh"
#include "ops.cuh"

namespace b200 {

// From this token count on.  It is faster from 100 tokens on (us, CUDA cores / here, 24 heads over 4: 192 37.5 / 22.6, 224 47.9 / 27.0, 300 85.6 / 31.0, 511 146 / 44.4), but of short rows
// the CUDA cores' sums are the more exact ones for some inputs: here products of small weights are cut off against the large ones, and scores are a few sums more.  Relative error against 64
// bits, 1e-7, CUDA cores / here (24 heads over 4):
//   tokens                                  224            320            511            1000           2047
//   normal values                           1.62 / 1.50    1.80 / 1.53    2.08 / 1.58    2.62 / 1.65    3.42 / 1.72
//   q 4 times as large                      2.88 / 2.82    3.19 / 2.96    3.64 / 3.13    4.47 / 3.37    5.70 / 3.65
//   v of one sign                           1.67 / 1.07    1.96 / 1.09    2.43 / 1.11    3.36 / 1.17    4.78 / 1.26
//   v of one sign, q 2 times as large       1.77 / 2.02    2.05 / 2.07    2.51 / 2.11    3.42 / 2.16    4.82 / 2.18
//   v of one sign, q 4 times as large       2.21 / 3.29    2.65 / 3.40    3.57 / 3.50    6.34 / 3.61    13.2 / 3.65
//   q 16 times as large                     4.22 / 4.86    4.54 / 5.17    4.86 / 5.48    5.21 / 5.86    5.63 / 6.30
// From 500 tokens on all but the last are better here; those scores (some tens, where the softmax of most rows sits on one or two keys) do not turn.  (What the score's last additions round off,
// kept and added in front of the exponential: q 16 times as large 224 3.93, 511 4.33, at a tenth of the time; v of one sign 3.22 and 3.42 all the same.)
constexpr int ATC_MIN_TOKENS = 512;
constexpr int ATC_M = 128, ATC_KEYS = 64, ATC_WARPS = 16, ATC_THREADS = ATC_WARPS * 32;
constexpr int ATC_CHUNK = 128 * 128;                         // bytes of 128 rows x 64 fp16
constexpr int ATC_PLANES = 4 * ATC_CHUNK;                    // q high; k high + low; v high + low: 64 KB each
constexpr int ATC_SMEM_BYTES = 1024 + 3 * ATC_PLANES + (2 * ATC_KEYS + 2 * ATT_D + 4 * ATC_M) * 4 + 64;
// tile image in global memory: k planes, v planes, 2^-s of the 64 keys, 2^-s of the 256 dims, the tile's range (magnitude bits: largest k,
// largest v, smallest of the keys' largest v; a key of zeros has none)
constexpr int ATC_IMG_KF = 2 * ATC_PLANES, ATC_IMG_VF = ATC_IMG_KF + ATC_KEYS * 4, ATC_IMG_RANGE = ATC_IMG_VF + ATT_D * 4;
constexpr int ATC_IMG_BYTES = 2 * ATC_PLANES + 2048;
constexpr uint32_t ATC_COL_O = 0, ATC_COL_S = 256, ATC_COL_QL = 384;
constexpr uint32_t ATC_HUGE = (127u + 60u) << 23;            // bits of 2^60
constexpr uint32_t ATC_TINY = (127u - 100u) << 23;           // bits of 2^-100: a dim of v all below it is past the shift's cap
constexpr uint32_t ATC_NONE = 0x7FFFFFFFu;
// The tensor core cuts the last bits of a sum of weights x v off, a step of 16 keys at a time.  What is missing in the mean (24 heads over 4, normal values, least squares
// against 64 bits, 1e-7 of the output): rows of 1 key 0.0, 2 0.4, 3 - 16 0.6, 17 - 32 1.0, 33 - 64 1.35, 1024 - 2048 1.55 (of positive v 0.0, 0.4, 0.5, 0.8, 1.65, 2.1; of queries a
// twentieth as large 0.0, 0.35, 0.4, 0.6, 0.85, 0.9); long rows whose softmax sits on one key, to 2^-6 of it, 0 - 0.5.  So a row's output is one unit in the last place larger where it sees
// more than 16 keys and its weights add up to more than that.  Relative error of a prompt, without / for every row / as here: normal 256 tokens 1.82e-7 / 1.57e-7 / 1.51e-7, 2047
// 2.09e-7 / 1.74e-7 / 1.72e-7; positive v 2.23e-7 / 1.21e-7 / 1.26e-7; of a row of one key 4.3e-8 / 1.24e-7 / 4.3e-8.  (The scores' sums, short as they are, need none: with 4e-8 to 1e-7
// more of them 1.70e-7 - 1.73e-7.)
constexpr float ATC_LIFT = 1.0f + 0x1p-23f, ATC_LIFT_WEIGHTS = 1.0f + 0x1p-6f;
constexpr int ATC_LIFT_KEYS = 17;
constexpr int ATC_V_RANGE = 12;                              // log2
constexpr float ATC_QK_RANGE = 4096.0f;
constexpr int ATC_REDO_QUERIES = ATC_WARPS * ATT_QPW;
static_assert(att_smem_bytes(ATC_WARPS) <= 3 * ATC_PLANES, "attn_simt reuses the planes");

__host__ __device__ constexpr uint32_t atc_idesc(int n) { return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(ATC_M >> 4) << 24); }

template <uint32_t IDESC>
__device__ __forceinline__ void atc_mma_ss(uint32_t d, uint32_t a_lo, uint32_t b_lo) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        ".reg .b64 da, db;\n\t"
        "mov.b64 da, {%1, %4};\n\t"
        "mov.b64 db, {%2, %4};\n\t"
        "setp.ne.b32 p, 1, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, {%5, %5, %5, %5}, p;\n\t"
        "}\n"
        ::"r"(d), "r"(a_lo), "r"(b_lo), "r"(IDESC), "r"(T16_DESC_HI), "r"(0u)
        : "memory");
}
__device__ __forceinline__ void tc_st8(uint32_t taddr, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n"
                 ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
__device__ __forceinline__ uint32_t atc_abs_bits(float x) { return __float_as_uint(x) & 0x7FFFFFFFu; }
// s with 2^14 <= max * 2^s < 2^15, at most `cap` (smaller maxima end lower: their products are that much smaller too)
__device__ __forceinline__ int atc_shift(uint32_t max_bits, int cap) { return min(cap, 141 - (int)(max_bits >> 23)); }
__device__ __forceinline__ float atc_pow2(int e) { return __uint_as_float((uint32_t)(127 + e) << 23); }
__device__ __forceinline__ void atc_split8(const float *x, float sc, uint4 &hi, uint4 &lo) {
    split_f16x2(__fmul_rn(x[0], sc), __fmul_rn(x[1], sc), hi.x, lo.x);
    split_f16x2(__fmul_rn(x[2], sc), __fmul_rn(x[3], sc), hi.y, lo.y);
    split_f16x2(__fmul_rn(x[4], sc), __fmul_rn(x[5], sc), hi.z, lo.z);
    split_f16x2(__fmul_rn(x[6], sc), __fmul_rn(x[7], sc), hi.w, lo.w);
}

// Whether a CTA's values range too widely for the planes (magnitude bits: largest scaled q, largest k, largest v, smallest of the
// keys' largest v, over every key that the CTA's tiles hold).
//   scores   a plane pair is off by at most 2^-40 of its row's largest value (2^-41 in the mean), times the other row's value: with
//            max |q| max |k| <= 2^12 the 512 products of a score add up to an error of about 2^-25, less than an fp32 sum's.
//            (Scores of that size do not occur: one channel alone would reach 4096.)
//   outputs  a key's weighted v is off by at most 2^-39 of the largest v, whatever its weight; a row's own largest output is no
//            smaller than the smallest key: within 2^12 of each other 1000 such errors add up to 2^-22 of it.
// Each range alone to 2^30 cost rows 1e-3 of their size (v) and scores 5e-4 (k); as it is every case of
// tests/test_gpu_prompt_attention.py is as exact as on the CUDA cores.  The ranges are looked at per CTA and not per row: both
// sides of the line are right, which of them a row takes does not matter.
__device__ __forceinline__ bool atc_too_wide(uint32_t q, uint32_t k, uint32_t v, uint32_t v_small) {
    if (max(q, max(k, v)) >= ATC_HUGE) return true;
    if (__fmul_rn(__uint_as_float(q), __uint_as_float(k)) > ATC_QK_RANGE) return true;
    return v_small != ATC_NONE && (int)(v >> 23) - (int)(v_small >> 23) > ATC_V_RANGE;
}

constexpr int ATC_PREP_THREADS = 256;
// grid (tiles, kv heads, 2): z 0 = k (warp = eight keys, lane = eight dims), z 1 = v (thread = one dim, all 64 keys).  Bound
// by latency: 16 MB in, 17 MB out at 2048 tokens.
__global__ void __launch_bounds__(ATC_PREP_THREADS) attn_planes_kernel(const float *k, const float *v, uint8_t *images, int n_tok, int n_head_kv) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int j0 = (int)blockIdx.x * ATC_KEYS, kvh = blockIdx.y;
    uint8_t *img = images + ((size_t)kvh * gridDim.x + blockIdx.x) * ATC_IMG_BYTES;
    uint32_t *range = reinterpret_cast<uint32_t *>(img + ATC_IMG_RANGE);
    __shared__ uint32_t top[ATC_PREP_THREADS / 32][ATC_KEYS];
    pdl_wait_prior_grid();
    pdl_launch_dependents();
    if (blockIdx.z == 0) {
        constexpr int ROWS = ATC_KEYS / (ATC_PREP_THREADS / 32);
        float x[ROWS][8];
        uint32_t seen = 0;
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            const int key = ROWS * warp + r;
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
            if (j0 + key < n_tok) {
                const float4 *src = reinterpret_cast<const float4 *>(k + ((size_t)(j0 + key) * n_head_kv + kvh) * ATT_D + 8 * lane);
                a = src[0];
                b = src[1];
            }
            x[r][0] = a.x; x[r][1] = a.y; x[r][2] = a.z; x[r][3] = a.w; x[r][4] = b.x; x[r][5] = b.y; x[r][6] = b.z; x[r][7] = b.w;
        }
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            const int key = ROWS * warp + r;
            uint32_t m = 0;
#pragma unroll
            for (int e = 0; e < 8; ++e) m = max(m, atc_abs_bits(x[r][e]));
            m = __reduce_max_sync(0xffffffffu, m);
            seen = max(seen, m);
            const int s = atc_shift(m, 63);
            uint4 hi, lo;
            atc_split8(x[r], atc_pow2(s), hi, lo);
            uint8_t *dst = img + (lane >> 3) * ATC_CHUNK + key * 128 + (((lane & 7) ^ (key & 7)) * 16);
            *reinterpret_cast<uint4 *>(dst) = hi;
            *reinterpret_cast<uint4 *>(dst + ATC_KEYS * 128) = lo;
            if (lane == 0) reinterpret_cast<float *>(img + ATC_IMG_KF)[key] = atc_pow2(-s);
        }
        if (lane == 0) top[warp][0] = seen;
        __syncthreads();
        if (warp == 0) {
            const uint32_t m = __reduce_max_sync(0xffffffffu, top[lane & (ATC_PREP_THREADS / 32 - 1)][0]);
            if (lane == 0) range[0] = m;
        }
    } else {
        const int d = threadIdx.x;
        float x[ATC_KEYS];
        const float *src = v + ((size_t)j0 * n_head_kv + kvh) * ATT_D + d;
#pragma unroll
        for (int e = 0; e < ATC_KEYS; ++e) x[e] = j0 + e < n_tok ? src[(size_t)e * n_head_kv * ATT_D] : 0.0f;
        uint32_t seen = 0;
#pragma unroll
        for (int e = 0; e < ATC_KEYS; ++e) seen = max(seen, atc_abs_bits(x[e]));
        const int s = atc_shift(seen, 112);
        reinterpret_cast<float *>(img + ATC_IMG_VF)[d] = atc_pow2(-s - 14);          // (and the weights' 2^-14)
#pragma unroll
        for (int g = 0; g < ATC_KEYS / 8; ++g) {
            uint4 hi, lo;
            atc_split8(x + 8 * g, atc_pow2(s), hi, lo);
            uint8_t *dst = img + ATC_PLANES + d * 128 + ((g ^ (d & 7)) * 16);
            *reinterpret_cast<uint4 *>(dst) = hi;
            *reinterpret_cast<uint4 *>(dst + 2 * ATC_CHUNK) = lo;
        }
        // the keys' largest values: over the warp's 32 dims (lane e keeps keys e and e + 32), then over the warps
        uint32_t own[2] = {0u, 0u};
#pragma unroll
        for (int e = 0; e < ATC_KEYS; ++e) {
            const uint32_t m = __reduce_max_sync(0xffffffffu, atc_abs_bits(x[e]));
            if (lane == (e & 31)) own[e >> 5] = m;
        }
        top[warp][lane] = own[0];
        top[warp][lane + 32] = own[1];
        const int tiny = __syncthreads_or(seen > 0u && seen < ATC_TINY ? 1 : 0);
        if (warp == 0) {
#pragma unroll
            for (int w = 0; w < ATC_PREP_THREADS / 32; ++w)
#pragma unroll
                for (int h = 0; h < 2; ++h) own[h] = max(own[h], top[w][lane + 32 * h]);
            const uint32_t most = __reduce_max_sync(0xffffffffu, max(own[0], own[1]));
            const uint32_t least = __reduce_min_sync(0xffffffffu, min(own[0] ? own[0] : ATC_NONE, own[1] ? own[1] : ATC_NONE));
            if (lane == 0) {
                range[1] = tiny ? ATC_NONE : most;
                range[2] = least;
            }
        }
    }
}

// Cold path, a call of its own so that it takes no registers from the kernel.
__device__ __noinline__ void attn_redo(float *smem, const float *q, const float *k, const float *v, float *out, int first, int head, int n_tok,
                                       int n_head, int n_head_kv, float scale) {
    for (int q0 = first; q0 < min(n_tok, first + ATC_M); q0 += ATC_REDO_QUERIES) {
        __syncthreads();
        attn_simt<ATC_WARPS>(smem, q, k, v, out, q0, head, n_tok, n_head, n_head_kv, scale);
    }
}

// grid: query blocks x heads, the longest rows of keys first (block index / n_head counts from the last query block)
__global__ void __launch_bounds__(ATC_THREADS, 1) attn_tc_kernel(const float *q, const float *k, const float *v, const uint8_t *images, float *out,
                                                                 int n_tok, int n_head, int n_head_kv, float scale) {
    extern __shared__ __align__(128) uint8_t smem[];
    uint8_t *qhi = smem + ((1024u - (smem_u32(smem) & 1023u)) & 1023u);
    uint8_t *kpl = qhi + ATC_PLANES, *vpl = kpl + ATC_PLANES;
    float *kf = reinterpret_cast<float *>(vpl + ATC_PLANES);             // [2][64] 2^-s of the tile's keys, tiles alternate
    float *vf = kf + 2 * ATC_KEYS;                                       // [2][256] 2^-s of the dims (and the weights' 2^-14)
    float *red = vf + 2 * ATT_D;                                         // [4][128] exchange between the four warps of a row
    uint64_t *qk = reinterpret_cast<uint64_t *>(red + 4 * ATC_M), *pv = qk + 1, *kfull = qk + 2, *vfull = qk + 3;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(vfull + 1);

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int cg = warp >> 2, row = 32 * (warp & 3) + lane;              // a thread's row, and its quarter of the row's columns
    const int qblocks = (n_tok + ATC_M - 1) / ATC_M;
    const int head = (int)blockIdx.x % n_head, first = (qblocks - 1 - (int)blockIdx.x / n_head) * ATC_M;
    const int kvh = head / (n_head / n_head_kv);
    const int query = first + row;
    const int ntiles = (min(n_tok, first + ATC_M) + ATC_KEYS - 1) / ATC_KEYS;
    const uint8_t *img = images + (size_t)kvh * ((n_tok + ATC_KEYS - 1) / ATC_KEYS) * ATC_IMG_BYTES;

    if (threadIdx.x == 0) {
        mbar_init(qk, 2);                                                // an arrival of each issuing warp
        for (int b = 1; b < 4; ++b) mbar_init(qk + b, 1);
        mbar_fence_init();
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // one thread each: the images of tile i
    auto load_k = [&](int i) {
        const uint64_t pol = policy_evict_last_or_default();
        const uint8_t *src = img + (size_t)i * ATC_IMG_BYTES;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // the factors were read by ordinary loads
        mbar_expect_tx(kfull, ATC_PLANES + ATC_KEYS * 4);
        bulk_g2s(kf + (i & 1) * ATC_KEYS, src + ATC_IMG_KF, ATC_KEYS * 4, kfull, pol);
        bulk_g2s(kpl, src, ATC_PLANES, kfull, pol);
    };
    auto load_v = [&](int i) {
        const uint64_t pol = policy_evict_last_or_default();
        const uint8_t *src = img + (size_t)i * ATC_IMG_BYTES;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // the factors were read by ordinary loads
        mbar_expect_tx(vfull, ATC_PLANES + ATT_D * 4);
        bulk_g2s(vf + (i & 1) * ATT_D, src + ATC_IMG_VF, ATT_D * 4, vfull, pol);
        bulk_g2s(vpl, src + ATC_PLANES, ATC_PLANES, vfull, pol);
    };

    // ---- q: row of the thread, 64 dims; high plane to shared memory, low plane to tensor memory.  (The launch this one may
    // run beside is attn_planes_kernel, which does not write q.)
    // Queries and outputs pass through shared memory (the planes' of k and v, a warp's 32 rows of 64 values each, 16-byte pieces swizzled), where a row's
    // values become a thread's: 512 bytes of two rows per access.  (A row per thread, 16 bytes of 32 rows per access: 12 us of a CTA's time in front of its
    // tiles and 7 behind them, where a tile takes 4.)
    float4 *box = reinterpret_cast<float4 *>(kpl) + warp * 512;
    const int row0 = first + 32 * (warp & 3);
    float qf;
    uint32_t seen;                                                       // magnitude bits of the row's largest q
    {
        float x[64];
        uint32_t m = 0;
        if ((reinterpret_cast<uintptr_t>(q) & 15u) == 0) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const int r = 2 * i + (lane >> 4), c = lane & 15;
                if (row0 + r < n_tok) cp_async16(box + r * 16 + (c ^ (r & 15)), q + ((size_t)(row0 + r) * n_head + head) * ATT_D + 64 * cg + 4 * c);
            }
            cp_async_commit();
            cp_async_wait<0>();
            __syncwarp();
#pragma unroll
            for (int c = 0; c < 16; ++c) {
                const float4 a = query < n_tok ? box[lane * 16 + (c ^ (lane & 15))] : make_float4(0.f, 0.f, 0.f, 0.f);
                x[4 * c] = a.x; x[4 * c + 1] = a.y; x[4 * c + 2] = a.z; x[4 * c + 3] = a.w;
            }
        } else {
            const float *src = q + ((size_t)query * n_head + head) * ATT_D + 64 * cg;
#pragma unroll
            for (int e = 0; e < 64; ++e) x[e] = query < n_tok ? src[e] : 0.0f;
        }
#pragma unroll
        for (int e = 0; e < 64; ++e) {
            x[e] = __fmul_rn(x[e], scale);
            m = max(m, atc_abs_bits(x[e]));
        }
        uint32_t *redu = reinterpret_cast<uint32_t *>(red);
        redu[cg * ATC_M + row] = m;
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < 4; ++c) m = max(m, redu[c * ATC_M + row]);
        seen = m;
        const int s = atc_shift(m, 63);
        qf = atc_pow2(-s);
        uint32_t lo32[32];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            uint4 hi, lo;
            atc_split8(x + 8 * j, atc_pow2(s), hi, lo);
            *reinterpret_cast<uint4 *>(qhi + cg * ATC_CHUNK + row * 128 + ((j ^ (row & 7)) * 16)) = hi;
            lo32[4 * j] = lo.x; lo32[4 * j + 1] = lo.y; lo32[4 * j + 2] = lo.z; lo32[4 * j + 3] = lo.w;
        }
        tc_st32(*tmem_slot + ((uint32_t)(32 * (warp & 3)) << 16) + ATC_COL_QL + (uint32_t)(32 * cg), lo32);
    }
    const uint32_t tmem = *tmem_slot;
    const uint32_t tlane = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
    // The tensor core's instructions, one elected lane of warp 0 or 1 (the code stays warp-uniform).  Products with a low plane
    // come first: the accumulator is small while they are added.
    // One sum of the scores: 16-dim steps n0 .. n0 + STEPS - 1 into 64 columns at d.
    auto sum_of = [&](uint32_t d, auto n0c, auto stepsc) {
        constexpr int N0 = decltype(n0c)::value, STEPS = decltype(stepsc)::value;
        constexpr uint32_t LOW = (ATC_KEYS * 128) >> 4;
        const uint32_t a0 = tc16_desc_lo(smem_u32(qhi)), b0 = tc16_desc_lo(smem_u32(kpl)), ql = tmem + ATC_COL_QL;
        auto at = [](int n) { return (uint32_t)((n >> 2) * (ATC_CHUNK >> 4) + 2 * (n & 3)); };
        tc_mma_f16_ts<false>(d, ql + (uint32_t)(8 * N0), b0 + at(N0), atc_idesc(ATC_KEYS));
#pragma unroll
        for (int n = N0 + 1; n < N0 + STEPS; ++n) tc_mma_f16_ts<true>(d, ql + (uint32_t)(8 * n), b0 + at(n), atc_idesc(ATC_KEYS));
#pragma unroll
        for (int n = N0; n < N0 + STEPS; ++n) atc_mma_ss<atc_idesc(ATC_KEYS)>(d, a0 + at(n), b0 + LOW + at(n));
#pragma unroll
        for (int n = N0; n < N0 + STEPS; ++n) atc_mma_ss<atc_idesc(ATC_KEYS)>(d, a0 + at(n), b0 + at(n));
    };
    // Two warps issue the scores' products, half of the sums each: from one warp 16 dims take 39 (q low) or 55 cycles, and its chain of waits and
    // issues is not overlapped.  (One warp, a barrier for each half of the dims, waits polled back to back: 2048 tokens 287 us, 600 tokens 60.6;
    // with two 279 and 58.9, when queries and outputs still went by a row per thread.)
    auto issue_qk_a = [&] {                                              // dims 0 .. 63, two sums, into the score columns
        tc_fence_after();
        if (warp == 0) {
            if (elect_one()) sum_of(tmem + ATC_COL_S, std::integral_constant<int, 0>{}, std::integral_constant<int, 2>{});
        } else {
            if (elect_one()) sum_of(tmem + ATC_COL_S + ATC_KEYS, std::integral_constant<int, 2>{}, std::integral_constant<int, 2>{});
        }
        __syncwarp();
    };
    auto issue_qk_b = [&] {                                              // dims 64 .. 255, four sums, into the output columns; the commit covers the others too
        tc_fence_after();
        if (warp == 0) {
            if (elect_one()) {
                sum_of(tmem + ATC_COL_O, std::integral_constant<int, 4>{}, std::integral_constant<int, 3>{});
                sum_of(tmem + ATC_COL_O + ATC_KEYS, std::integral_constant<int, 7>{}, std::integral_constant<int, 3>{});
                tc_commit(qk);
            }
        } else {
            if (elect_one()) {
                sum_of(tmem + ATC_COL_O + 2 * ATC_KEYS, std::integral_constant<int, 10>{}, std::integral_constant<int, 3>{});
                sum_of(tmem + ATC_COL_O + 3 * ATC_KEYS, std::integral_constant<int, 13>{}, std::integral_constant<int, 3>{});
                tc_commit(qk);
            }
        }
        __syncwarp();
    };
    auto issue_pv = [&] {
        tc_fence_after();
        const uint32_t b0 = tc16_desc_lo(smem_u32(vpl)), ph = tmem + ATC_COL_S, pl = ph + 32u;
        if (elect_one()) {
#pragma unroll
            for (int n = 0; n < 12; ++n) {
                const uint32_t a = (n < 4 ? pl : ph) + (uint32_t)(8 * (n & 3));
                const uint32_t b = b0 + (uint32_t)((n >= 4 && n < 8 ? (2 * ATC_CHUNK) >> 4 : 0) + 2 * (n & 3));
                if (n == 0) tc_mma_f16_ts<false>(tmem + ATC_COL_O, a, b, atc_idesc(ATT_D));
                else tc_mma_f16_ts<true>(tmem + ATC_COL_O, a, b, atc_idesc(ATT_D));
            }
            tc_commit(pv);
        }
        __syncwarp();
    };

    pdl_wait_prior_grid();                                               // the images
    if (warp == 4 && lane == 0) {
        load_k(0);
        load_v(0);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");        // q high: written here, read by the tensor core
    tc_st_wait();
    tc_fence_before();
    __syncthreads();
    bool ok = true;
    if (warp < 2) {
        ok = mbar_wait_try(kfull, 0);
        issue_qk_a();
        issue_qk_b();
    }

    float acc[64];                                                       // row, dims 64 cg ..
#pragma unroll
    for (int e = 0; e < 64; ++e) acc[e] = 0.0f;
    float m_run = -INFINITY, l_run = 0.0f, alpha = 0.0f;                 // l_run: of the thread's 16 columns of every tile
    auto add_tile = [&](int par) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            int o[2][16];
            tc_ld16(tlane + ATC_COL_O + (uint32_t)(64 * cg + 32 * h), o[0]);
            tc_ld16(tlane + ATC_COL_O + (uint32_t)(64 * cg + 32 * h + 16), o[1]);
            tc_ld_wait();
#pragma unroll
            for (int e = 0; e < 32; e += 4) {
                const float4 f = *reinterpret_cast<const float4 *>(vf + par * ATT_D + 64 * cg + 32 * h + e);
                float *a = acc + 32 * h + e;
                const int *t = o[e >> 4] + (e & 15);
                a[0] = __fmaf_rn(__int_as_float(t[0]), f.x, __fmul_rn(a[0], alpha));
                a[1] = __fmaf_rn(__int_as_float(t[1]), f.y, __fmul_rn(a[1], alpha));
                a[2] = __fmaf_rn(__int_as_float(t[2]), f.z, __fmul_rn(a[2], alpha));
                a[3] = __fmaf_rn(__int_as_float(t[3]), f.w, __fmul_rn(a[3], alpha));
            }
        }
    };
    for (int i = 0; i < ntiles; ++i) {
        const int j0 = i * ATC_KEYS;
        const uint32_t par = (uint32_t)(i & 1);
        float s[16], mx = -INFINITY;
        ok = mbar_wait_both(kfull, par, qk, par) && ok;                  // (the first is long complete; it makes the copied factors visible)
        tc_fence_after();
        {
            // (eight columns at a time: sixteen of two sums beside the outputs and the scores were more registers than a thread has, and what is
            // spilled beside 200 KB of shared memory comes from L2: 2048 tokens 292 -> 286 us, 600 tokens 63.2 -> 61.6 us)
#pragma unroll
            for (uint32_t h = 0; h < 16; h += 8) {
                int a[8], b[8], c[8], d[8];
                tc_ld8(tlane + ATC_COL_S + h + (uint32_t)(16 * cg), a);
                tc_ld8(tlane + ATC_COL_S + ATC_KEYS + h + (uint32_t)(16 * cg), b);
                tc_ld8(tlane + ATC_COL_O + h + (uint32_t)(16 * cg), c);
                tc_ld8(tlane + ATC_COL_O + ATC_KEYS + h + (uint32_t)(16 * cg), d);
                tc_ld_wait();
                float t[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) t[e] = __fadd_rn(__fadd_rn(__int_as_float(a[e]), __int_as_float(b[e])), __fadd_rn(__int_as_float(c[e]), __int_as_float(d[e])));
                tc_ld8(tlane + ATC_COL_O + 2 * ATC_KEYS + h + (uint32_t)(16 * cg), a);
                tc_ld8(tlane + ATC_COL_O + 3 * ATC_KEYS + h + (uint32_t)(16 * cg), b);
                tc_ld_wait();
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const float f = __fmul_rn(qf, kf[par * ATC_KEYS + 16 * cg + (int)h + e]);
                    s[h + e] = j0 + 16 * cg + (int)h + e <= query ? __fmul_rn(__fadd_rn(t[e], __fadd_rn(__int_as_float(a[e]), __int_as_float(b[e]))), f) : -INFINITY;
                    mx = fmaxf(mx, s[h + e]);
                }
            }
        }
        red[cg * ATC_M + row] = mx;
        tc_fence_before();
        if (!__syncthreads_and(ok ? 1 : 0)) break;                       // (a wait ran out: the CTA leaves as a whole)
        tc_fence_after();                                                // every score has been read: the weights take their place
        // (a barrier's next phase is begun only when the whole CTA has waited for this one: a thread that came later than a
        // phase's successor would wait for a parity that has passed)
        if (warp == 4 && lane == 0 && i + 1 < ntiles) load_k(i + 1);
        float m_new = m_run;
#pragma unroll
        for (int c = 0; c < 4; ++c) m_new = fmaxf(m_new, red[c * ATC_M + row]);
        alpha = expf(__fsub_rn(m_run, m_new));
        m_run = m_new;
        {
            uint32_t hi[8], lo[8];
            float sum = 0.0f;
#pragma unroll
            for (int e = 0; e < 16; e += 2) {
                const float p0 = expf(__fsub_rn(s[e], m_new)), p1 = expf(__fsub_rn(s[e + 1], m_new));
                sum = __fadd_rn(sum, __fadd_rn(p0, p1));
                split_f16x2(__fmul_rn(p0, 16384.0f), __fmul_rn(p1, 16384.0f), hi[e >> 1], lo[e >> 1]);
            }
            l_run = __fadd_rn(__fmul_rn(l_run, alpha), sum);
            tc_st8(tlane + ATC_COL_S + (uint32_t)(8 * cg), hi);
            tc_st8(tlane + ATC_COL_S + (uint32_t)(32 + 8 * cg), lo);
        }
        tc_st_wait();
        ok = mbar_wait_try(vfull, par) && ok;                            // in front of the CTA's barrier: load_v below begins the next phase
        tc_fence_before();
        __syncthreads();
        if (warp == 0) issue_pv();
        ok = mbar_wait_try(pv, par) && ok;
        tc_fence_after();
        if (i + 1 < ntiles) {
            if (warp == 4 && lane == 0) load_v(i + 1);
            if (warp < 2) {
                ok = mbar_wait_try(kfull, par ^ 1u) && ok;
                issue_qk_a();
            }
        }
        add_tile((int)par);
        if (i + 1 < ntiles) {
            tc_fence_before();
            __syncthreads();                                             // the output columns have been read: scores may go there
            if (warp < 2) issue_qk_b();
        }
    }
    __syncthreads();
    red[cg * ATC_M + row] = l_run;
    tc_fence_before();
    uint32_t k_most = 0, v_most = 0, v_least = ATC_NONE;
    for (int t = threadIdx.x; t < ntiles; t += ATC_THREADS) {
        const uint32_t *range = reinterpret_cast<const uint32_t *>(img + (size_t)t * ATC_IMG_BYTES + ATC_IMG_RANGE);
        k_most = max(k_most, range[0]);
        v_most = max(v_most, range[1]);
        v_least = min(v_least, range[2]);
    }
    uint4 *ranges = reinterpret_cast<uint4 *>(kf);                       // a warp each; every tile's factors have been read
    seen = __reduce_max_sync(0xffffffffu, seen);
    k_most = __reduce_max_sync(0xffffffffu, k_most);
    v_most = __reduce_max_sync(0xffffffffu, v_most);
    v_least = __reduce_min_sync(0xffffffffu, v_least);
    if (lane == 0) ranges[warp] = make_uint4(seen, k_most, v_most, v_least);
    __syncthreads();
    const uint4 r = ranges[lane & (ATC_WARPS - 1)];
    const bool redo = atc_too_wide(__reduce_max_sync(0xffffffffu, r.x), __reduce_max_sync(0xffffffffu, r.y), __reduce_max_sync(0xffffffffu, r.z),
                                   __reduce_min_sync(0xffffffffu, r.w));
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
    if (redo) {
        attn_redo(reinterpret_cast<float *>(qhi), q, k, v, out, first, head, n_tok, n_head, n_head_kv, scale);
        return;
    }
    const float l = __fadd_rn(__fadd_rn(red[row], red[ATC_M + row]), __fadd_rn(red[2 * ATC_M + row], red[3 * ATC_M + row]));
    const float inv = __fdiv_rn(query + 1 >= ATC_LIFT_KEYS && l >= ATC_LIFT_WEIGHTS ? ATC_LIFT : 1.0f, l);
    if ((reinterpret_cast<uintptr_t>(out) & 15u) == 0) {
#pragma unroll
        for (int c = 0; c < 16; ++c)
            box[lane * 16 + (c ^ (lane & 15))] = make_float4(__fmul_rn(acc[4 * c], inv), __fmul_rn(acc[4 * c + 1], inv), __fmul_rn(acc[4 * c + 2], inv), __fmul_rn(acc[4 * c + 3], inv));
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int r = 2 * i + (lane >> 4), c = lane & 15;
            if (row0 + r < n_tok) *reinterpret_cast<float4 *>(out + ((size_t)(row0 + r) * n_head + head) * ATT_D + 64 * cg + 4 * c) = box[r * 16 + (c ^ (r & 15))];
        }
    } else if (query < n_tok) {
        float *dst = out + ((size_t)query * n_head + head) * ATT_D + 64 * cg;
#pragma unroll
        for (int e = 0; e < 64; ++e) dst[e] = __fmul_rn(acc[e], inv);
    }
}

}  // namespace b200
