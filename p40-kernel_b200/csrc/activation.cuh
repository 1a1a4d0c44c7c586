// activation.cuh -- FWHT-1024 rotation and the Q8_1 quantiser (activation side of the path).
//
// Replaces, for sm_100a: fwht_1024_p40_kernel (src/kernels/elementwise_p40.cu:17-41) and
// quant_q8_1_pq2_kernel (src/kernels/gemv_p40.cu:168-196).  Output bytes follow the reference's
// HOST functions: fwht_blocks (src/fwht.h:20-42) and quantize_row_q8_1(..., permute = true)
// (src/pq2_0.h:99-126).
//
// A decode vector is a handful of latency-bound warps (<= 70 KB in, <= 20 KB out), a prompt's batch is bound by issue:
//   * rotation: a CTA per 1024-block with a warp per slice of 128 for few blocks, a warp per block (32 values per lane in
//     registers) for many; the ten butterfly stages run in the host's order (h = 1, 2, ..., 512), each output produced by
//     exactly one a + b or a - b with a the lower-index operand, so the fp32 bits equal the host's in either form;
//   * quantiser: eight lanes per 32-chunk, four values per lane (the same register layout the
//     rotation leaves behind, which is what lets the two fuse without a shuffle stage between).
#pragma once

#include "common.cuh"

namespace b200 {

// ---- quantiser core: 8 consecutive lanes own one 32-chunk, lane g (0..7) holds x[4g..4g+3] ----
// Returns through `word` the Q8_1 data word this lane stores (word index g of qs) and through
// `header` the d|s word (valid on every lane of the group).
// LONG: rounding in the longer form, the same values (list launch: round_ties_away_long).
template <bool LONG = false>
__device__ __forceinline__ void quantise_chunk_8lanes(const float (&v)[4], int lane, uint32_t &word, uint32_t &header) {
    float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    const float d = __fdiv_rn(amax, 127.0f);
    const float id = d > 0.0f ? __fdiv_rn(1.0f, d) : 0.0f;
    int sum = 0;
    uint32_t packed = 0;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        int q = LONG ? round_ties_away_long(__fmul_rn(v[e], id)) : round_ties_away(__fmul_rn(v[e], id));
        q = max(-127, min(127, q));
        sum += q;
        packed |= ((uint32_t)q & 0xFFu) << (8 * e);
    }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    // 4x4 byte transpose among the four lanes of each half-group: element j = 4g + e lands at
    // position 16*(j>>4) + 4*(j&3) + ((j>>2)&3) = byte (g&3) of word 4*(g>>2) + e, so this lane
    // (word g) gathers byte (g&3) from the lanes of its half-group.
    const int m = lane & 3;
    const int base = lane & ~3;
    word = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint32_t other = __shfl_sync(0xffffffffu, packed, base + k);
        word |= ((other >> (8 * m)) & 0xFFu) << (8 * k);
    }
    header = f32_to_f16_bits_ties_away(d) | (((uint32_t)sum & 0xFFFFu) << 16);
}

// The same for N (up to eight) chunks of each eight lanes at once, the N chains side by side; lane g of the eight divides for chunk
// g alone.
template <int N, bool LONG = false>
__device__ __forceinline__ void quantise_chunks_8lanes(const float (&v)[N][4], int lane, uint32_t (&word)[N], uint32_t (&header)[N]) {
    static_assert(N >= 1 && N <= 8, "a lane of the eight per chunk");
    if constexpr (N == 1) {                 // nothing to share
        quantise_chunk_8lanes<LONG>(v[0], lane, word[0], header[0]);
    } else {
        float amax[N], mine;
#pragma unroll
        for (int k = 0; k < N; ++k) amax[k] = fmaxf(fmaxf(fabsf(v[k][0]), fabsf(v[k][1])), fmaxf(fabsf(v[k][2]), fabsf(v[k][3])));
#pragma unroll
        for (int o = 1; o < 8; o <<= 1)
#pragma unroll
            for (int k = 0; k < N; ++k) amax[k] = fmaxf(amax[k], __shfl_xor_sync(0xffffffffu, amax[k], o));
        mine = amax[0];
#pragma unroll
        for (int k = 1; k < N; ++k) mine = (lane & 7) == k ? amax[k] : mine;
        const float d = __fdiv_rn(mine, 127.0f);
        const float my_id = d > 0.0f ? __fdiv_rn(1.0f, d) : 0.0f;
        const uint32_t my_d16 = f32_to_f16_bits_ties_away(d);
        int sum[N];
        uint32_t packed[N], d16[N];
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const float id = __shfl_sync(0xffffffffu, my_id, (lane & ~7) + k);
            d16[k] = __shfl_sync(0xffffffffu, my_d16, (lane & ~7) + k);
            sum[k] = 0;
            packed[k] = 0;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                int q = LONG ? round_ties_away_long(__fmul_rn(v[k][e], id)) : round_ties_away(__fmul_rn(v[k][e], id));
                q = max(-127, min(127, q));
                sum[k] += q;
                packed[k] |= ((uint32_t)q & 0xFFu) << (8 * e);
            }
        }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1)
#pragma unroll
            for (int k = 0; k < N; ++k) sum[k] += __shfl_xor_sync(0xffffffffu, sum[k], o);
        // the 4x4 byte transpose of quantise_chunk_8lanes
        const int m = lane & 3, base = lane & ~3;
#pragma unroll
        for (int k = 0; k < N; ++k) {
            word[k] = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t other = __shfl_sync(0xffffffffu, packed[k], base + j);
                word[k] |= ((other >> (8 * m)) & 0xFFu) << (8 * j);
            }
            header[k] = d16[k] | (((uint32_t)sum[k] & 0xFFFFu) << 16);
        }
    }
}

// Four consecutive floats: one 16-byte access when the caller's pointer allows it (VEC), else four 4-byte
// accesses -- the reference takes any float pointer (src/kernels/elementwise_p40.cu:75-80, gemv_p40.cu:200-208).
template <bool VEC>
__device__ __forceinline__ float4 load_f4(const float *p) {
    if (VEC) return *reinterpret_cast<const float4 *>(p);
    return make_float4(p[0], p[1], p[2], p[3]);
}
template <bool VEC>
__device__ __forceinline__ void store_f4(float *p, float4 v) {
    if (VEC) { *reinterpret_cast<float4 *>(p) = v; return; }
    p[0] = v.x; p[1] = v.y; p[2] = v.z; p[3] = v.w;
}

// One thread per four inputs.  X is [n_tok][n_in]; output block index = chunk * tok_stride + tok
// (tok_stride = 1 with n_tok = 1 gives the plain vector layout).
// EARLY: the next launch is let in at once (a mat-vec behind a vector's quantiser starts its weights: 5120 -> 1024 4.68 us the two, 4.90 by ending; the choice made here
// and not by the host: 4.80), else by ending (200 tokens of 5120 3.37 and 3.13).
template <bool VEC, bool EARLY>
__global__ void __launch_bounds__(256) quant_q8_1_kernel(const float *X, uint32_t *__restrict__ out,
                                                         int n_in, int n_tok) {
    pdl_wait_prior_grid();
    if (EARLY) pdl_launch_dependents();
    const int lane = threadIdx.x & 31;
    const int per_tok = n_in >> 2;
    const long long total = (long long)per_tok * n_tok;
    const long long stride = (long long)gridDim.x * blockDim.x;
    // whole warps iterate together: total is a multiple of 8 and a warp covers 32 threads
    for (long long i0 = (long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31); i0 < total; i0 += stride) {
        const long long i = i0 + lane;
        const bool live = i < total;
        const long long ic = live ? i : total - 1;
        const int tok = (int)(ic / per_tok);
        const int g4 = (int)(ic - (long long)tok * per_tok);
        const float4 f = load_f4<VEC>(X + (size_t)tok * n_in + 4 * (size_t)g4);
        const float v[4] = {f.x, f.y, f.z, f.w};
        uint32_t word, header;
        quantise_chunk_8lanes(v, lane, word, header);
        if (live) {
            const int chunk = g4 >> 3;
            uint32_t *blk = out + 9 * ((size_t)chunk * n_tok + tok);
            blk[1 + (lane & 7)] = word;
            if ((lane & 7) == 0) blk[0] = header;
        }
    }
}

// ---- rotation split over warps: one warp per 128-element slice ----------------------------------
// A 1024-block is eight slices r = 0..7 of 128 consecutive elements; lane l of the slice's warp holds
// elements 4l .. 4l+3.  The butterflies with h = 1 .. 64 stay inside a slice (front); those with
// h = 128, 256, 512 combine the eight slices element by element (back), through shared memory.  Every
// output is still produced by the host's a + b / a - b, stage by stage, so the bits are the same: a - b is
// computed as (-b) + a ... with IEEE addition that is the same rounding.
__device__ __forceinline__ void fwht_slice_front(float (&v)[4], int lane) {
    {
        const float a = v[0], b = v[1], c = v[2], d = v[3];
        const float s0 = __fadd_rn(a, b), s1 = __fsub_rn(a, b), s2 = __fadd_rn(c, d), s3 = __fsub_rn(c, d);
        v[0] = __fadd_rn(s0, s2); v[2] = __fsub_rn(s0, s2);
        v[1] = __fadd_rn(s1, s3); v[3] = __fsub_rn(s1, s3);
    }
#pragma unroll
    for (int s = 0; s < 5; ++s) {
        const bool upper = (lane >> s) & 1;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float mine = v[e];
            const float other = __shfl_xor_sync(0xffffffffu, mine, 1 << s);
            v[e] = upper ? __fsub_rn(other, mine) : __fadd_rn(mine, other);
        }
    }
}
// `block` points at the eight front-transformed slices of one 1024-block ([8][32] float4); returns
// slice r of the finished rotation (scaled by 1/32) for this lane.
__device__ __forceinline__ void fwht_slice_back(const float4 *block, int r, int lane, float (&out)[4]) {
    float a[8][4];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const float4 f = block[(r ^ j) * 32 + lane];
        a[j][0] = f.x; a[j][1] = f.y; a[j][2] = f.z; a[j][3] = f.w;
    }
    // the element at index q of a pair (q, q | h) becomes a_lower + a_upper, the upper one a_lower - a_upper;
    // with m = sign mask when this slice is the upper one:  new(q) = partner + (own ^ m)
    const uint32_t m0 = (r & 1) ? 0x80000000u : 0u, m1 = (r & 2) ? 0x80000000u : 0u, m2 = (r & 4) ? 0x80000000u : 0u;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        float u[4];      // h = 128 at slices r, r^2, r^4, r^6
#pragma unroll
        for (int k = 0; k < 4; ++k)
            u[k] = __fadd_rn(a[2 * k + 1][e], __uint_as_float(__float_as_uint(a[2 * k][e]) ^ m0));
        // h = 256 at slices r (u[0] with u[1]) and r^4 (u[2] with u[3])
        const float w0 = __fadd_rn(u[1], __uint_as_float(__float_as_uint(u[0]) ^ m1));
        const float w1 = __fadd_rn(u[3], __uint_as_float(__float_as_uint(u[2]) ^ m1));
        // h = 512 at slice r
        out[e] = __fmul_rn(__fadd_rn(w1, __uint_as_float(__float_as_uint(w0) ^ m2)), 0.03125f);
    }
}

// One CTA per 1024-block, one warp per slice: n_tok * (n_in / 1024) CTAs.  Bound by latency: a warp that did a whole block
// alone issued eight times as much in one serial chain (a vector of 5120: 7.2 us against 3.4 us with the launch).  X [n_tok][n_in] read-only;
// x_rot (nullable, may alias X) receives the rotated values; xq (nullable) the Q8_1 blocks at chunk * n_tok + tok.
constexpr int FWHT_THREADS = 256;
template <bool VEC>
__global__ void __launch_bounds__(FWHT_THREADS) fwht_quant_kernel(const float *X, const float *signs, float *x_rot, uint32_t *xq, int n_in, int n_tok) {
    __shared__ float4 front[FWHT_N / 4];
    const int lane = threadIdx.x & 31, r = threadIdx.x >> 5;
    const int blocks_per_tok = n_in / FWHT_N;
    const int tok = (int)blockIdx.x / blocks_per_tok, blk = (int)blockIdx.x - tok * blocks_per_tok;
    const size_t base = (size_t)tok * n_in + (size_t)blk * FWHT_N + r * 128 + 4 * lane;
    pdl_wait_prior_grid();
    pdl_launch_dependents();
    const float4 f = load_f4<VEC>(X + base);
    float v[4] = {f.x, f.y, f.z, f.w};
    if (signs) {
        const float4 s = load_f4<VEC>(signs + (size_t)blk * FWHT_N + r * 128 + 4 * lane);
        v[0] = __fmul_rn(v[0], s.x); v[1] = __fmul_rn(v[1], s.y);
        v[2] = __fmul_rn(v[2], s.z); v[3] = __fmul_rn(v[3], s.w);
    }
    fwht_slice_front(v, lane);
    front[threadIdx.x] = make_float4(v[0], v[1], v[2], v[3]);
    __syncthreads();
    fwht_slice_back(front, r, lane, v);
    if (x_rot) store_f4<VEC>(x_rot + base, make_float4(v[0], v[1], v[2], v[3]));
    if (xq) {
        uint32_t word, header;
        quantise_chunk_8lanes(v, lane, word, header);
        const int chunk = blk * 32 + r * 4 + (lane >> 3);
        uint32_t *dst = xq + 9 * ((size_t)chunk * n_tok + tok);
        dst[1 + (lane & 7)] = word;
        if ((lane & 7) == 0) dst[0] = header;
    }
}

// The same, a warp per block: fewer instructions a block, a longer chain.  Bound by instruction issue and by the pipe that shuffles and shared memory
// have in common.  Element 32 c + p of the block: the butterflies with h = 1 .. 16 run with four values of a lane's, by shuffles over eight lanes; then c is
// the register and p the lane (through shared memory) for h = 32 .. 512; then a lane has a chunk to itself, whose maximum, sum and words need no other lane.
// (32 values of a lane's all the way, every exchange a shuffle, 256 of them a block, four warps a CTA, us: 2000 blocks with quantiser 5.82 -> 4.65, 5000 10.55 ->
// 8.50, 10000 17.8 -> 14.4, stored as well 19.4 -> 16.9; rotation alone 900 2.84 -> 2.46, 10000 11.7 both.)
constexpr int FWHT_ROW = 36;           // words a row of 32: 16-byte accesses of eight rows, and 4-byte ones of any, meet no bank twice
template <bool VEC>
__global__ void __launch_bounds__(32, 32) fwht_quant_warp_kernel(const float *X, const float *signs, float *x_rot, uint32_t *xq, int n_in, int n_tok) {
    __shared__ __align__(16) float sm[32 * FWHT_ROW];
    const int lane = threadIdx.x;
    const int blocks_per_tok = n_in / FWHT_N;
    const int tok = (int)blockIdx.x / blocks_per_tok, blk = (int)blockIdx.x - tok * blocks_per_tok;
    const size_t base = (size_t)tok * n_in + (size_t)blk * FWHT_N;
    pdl_wait_prior_grid();
    float v[32];
    {
        float4 f[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) f[r] = load_f4<VEC>(X + base + r * 128 + 4 * lane);
        if (signs) {
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const float4 s = load_f4<VEC>(signs + (size_t)blk * FWHT_N + r * 128 + 4 * lane);
                f[r].x = __fmul_rn(f[r].x, s.x); f[r].y = __fmul_rn(f[r].y, s.y);
                f[r].z = __fmul_rn(f[r].z, s.z); f[r].w = __fmul_rn(f[r].w, s.w);
            }
        }
        const float2 minus = make_float2(-1.0f, -1.0f);
        float2 a[8], b[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) {           // h = 1, 2
            const float s0 = __fadd_rn(f[r].x, f[r].y), s1 = __fsub_rn(f[r].x, f[r].y), s2 = __fadd_rn(f[r].z, f[r].w), s3 = __fsub_rn(f[r].z, f[r].w);
            a[r] = add2(make_float2(s0, s1), make_float2(s2, s3));
            b[r] = fma2(make_float2(s2, s3), minus, make_float2(s0, s1));
        }
#pragma unroll
        for (int s = 0; s < 3; ++s) {           // h = 4, 8, 16: own + other, or other - own
            const float sign = (lane >> s) & 1 ? -1.0f : 1.0f;
            const float2 sign2 = make_float2(sign, sign);
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const float2 oa = make_float2(__shfl_xor_sync(0xffffffffu, a[r].x, 1 << s), __shfl_xor_sync(0xffffffffu, a[r].y, 1 << s));
                const float2 ob = make_float2(__shfl_xor_sync(0xffffffffu, b[r].x, 1 << s), __shfl_xor_sync(0xffffffffu, b[r].y, 1 << s));
                a[r] = fma2(a[r], sign2, oa);
                b[r] = fma2(b[r], sign2, ob);
            }
        }
#pragma unroll
        for (int r = 0; r < 8; ++r)
            *reinterpret_cast<float4 *>(sm + (4 * r + (lane >> 3)) * FWHT_ROW + 4 * (lane & 7)) = make_float4(a[r].x, a[r].y, b[r].x, b[r].y);
        __syncwarp();
        float2 z[16];                           // chunks 2 k and 2 k + 1
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const float lo = sm[2 * k * FWHT_ROW + lane], hi = sm[(2 * k + 1) * FWHT_ROW + lane];
            z[k] = make_float2(__fadd_rn(lo, hi), __fsub_rn(lo, hi));          // h = 32
        }
#pragma unroll
        for (int s = 0; s < 4; ++s)             // h = 64 .. 512
#pragma unroll
            for (int k = 0; k < 16; ++k)
                if (!((k >> s) & 1)) {
                    const float2 lo = z[k], hi = z[k | (1 << s)];
                    z[k] = add2(lo, hi);
                    z[k | (1 << s)] = fma2(hi, minus, lo);
                }
#pragma unroll
        for (int k = 0; k < 16; ++k) v[2 * k] = __fmul_rn(z[k].x, 0.03125f), v[2 * k + 1] = __fmul_rn(z[k].y, 0.03125f);
    }
    if (x_rot) {
#pragma unroll
        for (int c = 0; c < 32; ++c) x_rot[base + 32 * c + lane] = v[c];
    }
    if (!xq) return;
#pragma unroll
    for (int c = 0; c < 32; ++c) sm[c * FWHT_ROW + lane] = v[c];           // the words this lane has read
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const float4 f = *reinterpret_cast<const float4 *>(sm + lane * FWHT_ROW + 4 * j);
        v[4 * j] = f.x; v[4 * j + 1] = f.y; v[4 * j + 2] = f.z; v[4 * j + 3] = f.w;
    }
    float top[4] = {fabsf(v[0]), fabsf(v[1]), fabsf(v[2]), fabsf(v[3])};      // (not 0: of a chunk of NaN it is NaN)
#pragma unroll
    for (int i = 4; i < 32; ++i) top[i & 3] = fmaxf(top[i & 3], fabsf(v[i]));
    const float d = __fdiv_rn(fmaxf(fmaxf(top[0], top[1]), fmaxf(top[2], top[3])), 127.0f);
    const float id = d > 0.0f ? __fdiv_rn(1.0f, d) : 0.0f;
    uint32_t word[8];
    int sum = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {               // word 4 a + m: values 16 a + m, + 4, + 8, + 12
        word[i] = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int q = max(-127, min(127, round_ties_away(__fmul_rn(v[16 * (i >> 2) + (i & 3) + 4 * j], id))));
            word[i] |= ((uint32_t)q & 0xFFu) << (8 * j);
        }
        sum = __dp4a((int)word[i], 0x01010101, sum);
    }
    __syncwarp();                               // every row has been read
    uint32_t *out = reinterpret_cast<uint32_t *>(sm);
    out[9 * lane] = f32_to_f16_bits_ties_away(d) | (((uint32_t)sum & 0xFFFFu) << 16);
#pragma unroll
    for (int i = 0; i < 8; ++i) out[9 * lane + 1 + i] = word[i];
    __syncwarp();
    const int part = lane / 9;                  // three chunks of nine words at a time
    uint32_t *dst = xq + 9 * ((size_t)(blk * 32 + part) * n_tok + tok) + (lane - 9 * part);
    if (lane < 27) {
#pragma unroll
        for (int k = 0; k < 11; ++k)
            if (k < 10 || part < 2) dst[(size_t)k * 27 * n_tok] = out[27 * k + lane];
    }
}

}  // namespace b200
