// kv.cuh -- the growing Q8_0 K/V cache of the full-attention layers: append (quantise) and single-query decode
// attention over it.  Replaces, for sm_100a, src/kernels/kv_p40.cu:47-245 of the reference; the numeric core it
// follows is src/kv_cache.h:100-176 (Q8_0 rows: d = amax / 127, round to nearest with ties away, fp16 scale by the
// host's rule; score = int8 dot x both scales; split-K online softmax; merge of the splits).
//
// Layout (unchanged, it is the format, src/kv_cache.h:35-46): head-major, K and V separate,
// block[((layer * n_kv_head + kv_head) * capacity + pos) * 8 + blk], 34-byte blocks -- the 8 blocks of a position are
// 272 contiguous bytes, consecutive positions follow each other, so a run of positions of one (layer, kv head) is ONE
// contiguous, 16-byte aligned span.
//
// Decode on B200: one CTA per (kv head, split of the positions) serves the SIX query heads that share the kv head
// (grouped-query attention), so K and V cross HBM once per group, not once per query head; both products run on the
// tensor cores.  The query heads are quantised in the kernel's prologue (no separate launch, no buffer).
#pragma once

#include "common.cuh"

#include <type_traits>

namespace b200 {

constexpr int KV_D = 256, KV_NBLK = 8, KV_ROW = KV_NBLK * 34;      // 272 bytes per position and head
constexpr int KV_TILE = 64;                                          // positions per tile
constexpr int KV_MAX_GROUP = 8;                                      // query heads per kv head the kernel is built for

// ---- Q8_0 row quantiser: 4 lanes per 32-value block, 8 values per lane ---------------------------------------------
// Bytes equal kv_quantize_row_q8_0 (src/kv_cache.h:100-117).  (The reference's device kernels give a lane 4 values,
// which covers only half of every block, src/kernels/kv_p40.cu:47-51,72; the host function is the one followed.)
__device__ __forceinline__ float kv_amax_8(const float (&x)[8]) {
    float amax = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(x[i]));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    return fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
}
__device__ __forceinline__ void kv_words_8(const float (&x)[8], float id, uint32_t (&word)[2]) {
    word[0] = word[1] = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        int v = round_ties_away(__fmul_rn(x[i], id));
        v = max(-127, min(127, v));
        word[i >> 2] |= ((uint32_t)v & 0xFFu) << (8 * (i & 3));
    }
}
// One warp per (token, kv head) row of K and of V: lane = (block lane / 4, eight dims).
// EARLY: the rows are asked into L2 while the launch before this one still runs (L2 hands out what it finds at the load, whoever writes
// in between), an aligned row by one bulk request.  That pays while the grid is resident at once: blocks that start later have no wait to
// hide it in.  16 layers in us (rows stored by halfwords, as then), without / by lines / as here; inputs not in L2: 512 tokens 61.4 / 55.3 / 53.3, 1024 88.0 / 79.9 / 77.8, 4096
// 178.2 / 182.3 / without; inputs in L2: 64 tokens 33.2 / 33.0 / 33.0, 512 44.5 / 49.4 / 46.9, 1024 80.2 / 74.7 / 74.0, 4096 172.5 / 176.4 /
// without.  Stored as now, by calls, without / as here: 1 token 23.6 / 22.3, 200 37.4 / 33.3, 512 50.2 / 43.2, 1024 80.0 / 70.5, 2048 104.4 / 99.2.  (The first tiles of the attention below, asked for likewise: no gain.)
constexpr int KV_APPEND_WARPS = 8;
template <bool VEC, bool EARLY>
__global__ void __launch_bounds__(32 * KV_APPEND_WARPS) kv_append_kernel(uint8_t *K, uint8_t *V,
                                                        const float *ksrc, const float *vsrc,
                                                        int pos0, int n_tok, int n_kv_head, int capacity, int layer) {
    __shared__ __align__(16) uint8_t rows[KV_APPEND_WARPS][2][KV_ROW];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int row = blockIdx.x * KV_APPEND_WARPS + warp;                        // token * n_kv_head + head
    if (row >= n_tok * n_kv_head) return;
    const int tok = row / n_kv_head, h = row - tok * n_kv_head;
    const int blk = lane >> 2, sub = lane & 3;
    const size_t base = (((size_t)layer * n_kv_head + h) * capacity + (size_t)(pos0 + tok)) * KV_ROW;
    const float *kr = ksrc + (size_t)row * KV_D + blk * 32 + sub * 8;
    const float *vr = vsrc + (size_t)row * KV_D + blk * 32 + sub * 8;
    float kx[8], vx[8];
    if (EARLY && VEC) {
        if (lane == 0) {
            bulk_prefetch_l2(kr, KV_D * 4);
            bulk_prefetch_l2(vr, KV_D * 4);
        }
    } else if (EARLY && sub == 0) {
        prefetch_l2(kr);
        prefetch_l2(vr);
    }
    pdl_wait_prior_grid();
    pdl_launch_dependents();
    if (VEC) {
        const float4 a = *reinterpret_cast<const float4 *>(kr), b = *reinterpret_cast<const float4 *>(kr + 4);
        const float4 c = *reinterpret_cast<const float4 *>(vr), e = *reinterpret_cast<const float4 *>(vr + 4);
        kx[0] = a.x; kx[1] = a.y; kx[2] = a.z; kx[3] = a.w; kx[4] = b.x; kx[5] = b.y; kx[6] = b.z; kx[7] = b.w;
        vx[0] = c.x; vx[1] = c.y; vx[2] = c.z; vx[3] = c.w; vx[4] = e.x; vx[5] = e.y; vx[6] = e.z; vx[7] = e.w;
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) { kx[i] = kr[i]; vx[i] = vr[i]; }
    }
    // the divisions of K by the even lanes of the four, of V by the odd ones
    const float kmax = kv_amax_8(kx), vmax = kv_amax_8(vx), d = __fdiv_rn(sub & 1 ? vmax : kmax, 127.0f), id = d > 0.0f ? __fdiv_rn(1.0f, d) : 0.0f;
    const uint32_t d16 = f32_to_f16_bits_ties_away(d);
    uint32_t kw[2], vw[2];
    kv_words_8(kx, __shfl_sync(0xffffffffu, id, lane & ~3), kw);
    kv_words_8(vx, __shfl_sync(0xffffffffu, id, lane | 1), vw);
    // Blocks start on 2-byte boundaries, rows on 16-byte ones: a row is put together in shared memory by halfwords (scale, then this lane's 8 bytes) and
    // stored by 17 lanes.  (By halfwords to memory, five stores a row, each to all of its sectors, and with a division per lane and row: 16 layers, us, by
    // calls / as here: 1 token 25.0 / 22.3, 64 34.5 / 28.8, 512 51.5 / 43.2, 1024 89.7 / 70.5, 2048 103.8 / 99.0, 4096 176 / 170.5.)
    uint8_t *kb = rows[warp][0], *vb = rows[warp][1];
    unsigned short *kp = reinterpret_cast<unsigned short *>(kb + 34 * blk), *vp = reinterpret_cast<unsigned short *>(vb + 34 * blk);
    if (sub < 2) (sub ? vp : kp)[0] = (unsigned short)d16;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        kp[1 + 4 * sub + 2 * j] = (unsigned short)(kw[j] & 0xFFFFu); kp[2 + 4 * sub + 2 * j] = (unsigned short)(kw[j] >> 16);
        vp[1 + 4 * sub + 2 * j] = (unsigned short)(vw[j] & 0xFFFFu); vp[2 + 4 * sub + 2 * j] = (unsigned short)(vw[j] >> 16);
    }
    __syncwarp();
    if (lane < KV_ROW / 16) {
        const uint4 a = reinterpret_cast<const uint4 *>(kb)[lane], c = reinterpret_cast<const uint4 *>(vb)[lane];
        reinterpret_cast<uint4 *>(K + base)[lane] = a;
        reinterpret_cast<uint4 *>(V + base)[lane] = c;
    }
}

// ---- decode attention ----------------------------------------------------------------------------------------------
// One CTA = four warps, one split of the positions of one kv head, all query heads of its group; tiles of 64 positions.
//   scores   warp w = positions 16 w .. 16 w + 15 of the tile.  The int8 products of a 32-value block run on mma.sync
//            (m16n8k32: 16 positions x 8 heads, int32 sums, exact); the two scales are applied per block in fp32.  The
//            warp's 16 positions form a softmax step of their own: weights relative to the warp's maximum.
//   values   warp w = output dims 64 w .. 64 w + 63 (two V blocks), all 64 positions and all heads.  V bytes become fp16
//            exactly (int8 fits), a weight (softmax weight x the chunk's rescale x the V block's scale x a power of two)
//            is split into two fp16 planes, high and low (22 - 23 bits, the size of expf's own error), which are rows 0 - 7
//            and 8 - 15 of one m16n8k16: one instruction multiplies both planes, accumulators are fp32.  The planes hold
//            2^-39 of the largest V scale of the split and of the warp's two blocks; where scales lie further apart than
//            KV_V_RANGE, a second pass over the tile multiplies what they left.
// What bounded the kernel before was instruction issue (5860 warp instructions per 32 positions: fp32 multiply-adds of
// every value for every head on the CUDA cores; 1500 GB/s).  This form issues 2700, start and merge included.
//
// 34-byte blocks: two blocks are 17 words.  Of an even block words 1 .. 7 are eight-aligned code words and word 0's high
// and word 8's low half make the eighth ("slot 0" = values 0, 1, 30, 31, slot i = values 4 i - 2 .. 4 i + 1); the odd block's
// eight words start at word 9.  The order of values inside a block does not matter to a sum, so nothing is shifted.
//
// Splits: the CTAs of a cluster share one kv head; their (m, l, acc) meet through distributed shared memory, every CTA of
// the cluster merging one slice of the dims.  With more than one cluster per head the merged slices go to a workspace and
// the last cluster to arrive at a slice's counter adds them up and writes the output: one launch per call (the merge was
// a kernel of its own).  Clusters of 16 serve the lengths where they halve the tiles of a split (513 positions on) and where two
// clusters of eight would need the second merge (up to 3071).
//
// Up to 3071 positions, one cluster per kv head (PUSH), the kernel is a chain of latencies: 9400 cycles from the end of the launch in front to
// the output of 9 positions, 10500 of 701.  What that form does about them: eight warps (a warp has half of the dims of 16 scores, the halves meet
// through shared memory, and one V block), and every CTA sends its slices and its (m, l) to whom they concern, who counts the bytes on a barrier
// (behind ordinary stores, at the cluster's barrier, and read from there: 3500 cycles; now 1500).  PUSH = 1: splits of at most one tile, without the second buffer and
// what a loop carries.  16 layers with their appends, us, before -> now (four warps, merged by reading): 9 positions 116 -> 96, 131 121 -> 100, 701 131 ->
// 105, 1024 133 -> 106, 1101 147 -> 133, 3001 185 -> 171.  (PUSH = 2 at 701: 111.)
constexpr int KV_THREADS = 128, KV_WARPS = 4, KV_BUFS = 2, KV_CLUSTER = 8, KV_WIDE_CLUSTER = 16;
constexpr int KV_HALF_BYTES = KV_TILE * KV_ROW;                      // the K (or V) rows of a tile
constexpr int KV_WT_STRIDE = KV_TILE + 8;                            // weights of a head: 8 g + 2 t are 32 different banks
constexpr int KV_SLICE = KV_D / KV_CLUSTER;                          // output dims a CTA of the cluster merges
constexpr int KV_MAX_CLUSTERS = 64;                                  // per kv head
// Exponents between the largest V scale so far and the smallest (not zero) of a tile up to which two planes of a weight do: a position
// of full weight keeps 2^-26 of itself.  Past it a large scale without weight took bits from the others (1e6 among values of
// 0.06: 3e-6 of the output).  A scale below fp16's normal range counts as the smallest there is.
constexpr int KV_V_RANGE = 12;
constexpr int KV_REC = KV_MAX_GROUP * (KV_SLICE + 2);                // floats of a cluster's merged slice: acc, m, l
constexpr int KV_Q_STRIDE = 64 + 4;                                  // words of a quantised query head: 4 g + t are 32 different banks
constexpr int KV_TABLE_BYTES = 128 + KV_MAX_GROUP * KV_WT_STRIDE * 4 + 3 * KV_MAX_GROUP * 8 * 4 + KV_MAX_GROUP * KV_Q_STRIDE * 4;
constexpr int KV_SMEM_BYTES = KV_TABLE_BYTES + KV_BUFS * 2 * KV_HALF_BYTES;
constexpr int KV_PUSH_WARPS = 8;
constexpr int KV_PUSH_SMEM_BYTES = KV_TABLE_BYTES + KV_MAX_GROUP * KV_D * 4 + KV_WIDE_CLUSTER * KV_MAX_GROUP * 8 + KV_PUSH_WARPS * 32 * 16;
static_assert(16384 >= KV_MAX_GROUP * (KV_D + 2) * 4 && KV_BUFS * 2 * KV_HALF_BYTES >= 16384 + 3 * KV_MAX_CLUSTERS * KV_MAX_GROUP * 4, "the merge reuses the tile buffers");

__device__ __forceinline__ void mma_s8_16832(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}
__device__ __forceinline__ void mma_f16_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// (a, b) -> high plane and what is left of them, as fp16 pairs
__device__ __forceinline__ void split_f16x2(float a, float b, uint32_t &hi, uint32_t &lo) {
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(__fsub_rn(a, f.x), __fsub_rn(b, f.y));
    hi = *reinterpret_cast<const uint32_t *>(&h);
    lo = *reinterpret_cast<const uint32_t *>(&l);
}
// What the planes left of (a, b), times 2^24 (at most 2^-10 of a value below 2^14): together they hold 2^-63 of the largest.  Of an
// infinity nothing is left.
__device__ __forceinline__ void split_rest_f16x2(float a, float b, uint32_t &hi, uint32_t &lo) {
    const float2 h = __half22float2(*reinterpret_cast<const __half2 *>(&hi)), l = __half22float2(*reinterpret_cast<const __half2 *>(&lo));
    const float ra = __fsub_rn(__fsub_rn(a, h.x), l.x), rb = __fsub_rn(__fsub_rn(b, h.y), l.y);
    split_f16x2(fabsf(ra) < 1.0f ? __fmul_rn(ra, 0x1p24f) : 0.0f, fabsf(rb) < 1.0f ? __fmul_rn(rb, 0x1p24f) : 0.0f, hi, lo);
}
__device__ __forceinline__ float half_bits_lo(uint32_t w) { return f16_bits_to_f32(w & 0xFFFFu); }
__device__ __forceinline__ float half_bits_hi(uint32_t w) { return f16_bits_to_f32(w >> 16); }
__device__ __forceinline__ float ld_cluster_f32(const float *p, uint32_t rank) {
    uint32_t a;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}

// grid (n_split, n_kv_head), cluster (CL, 1, 1), n_split a multiple of CL (PUSH: CL, else CL is KV_CLUSTER); split s covers positions
// s * chunk .. min((s + 1) * chunk, pos + 1) - 1 (a split may be empty).  counters: one per (kv head, slice), zero before
// and after every launch.
template <int GRP, int CL = KV_CLUSTER, int PUSH = 0>
__global__ void __launch_bounds__(PUSH ? 32 * KV_PUSH_WARPS : KV_THREADS, PUSH ? 2 : 3) kv_attn_kernel(const float *q, const uint8_t *K, const uint8_t *V, float *ws, unsigned int *counters, float *out,
                                                                int pos, int chunk, int n_kv_head, int capacity, int layer, float scale) {
    static_assert(GRP <= KV_MAX_GROUP, "");
    constexpr int WARPS = PUSH ? KV_PUSH_WARPS : KV_WARPS, THREADS = 32 * WARPS;
    constexpr int NB = KV_NBLK / WARPS;                                          // V blocks of a warp
    extern __shared__ __align__(128) uint8_t smem[];
    uint64_t *kfull = reinterpret_cast<uint64_t *>(smem), *vfull = kfull + KV_BUFS, *met = vfull + KV_BUFS;
    uint8_t *raw = smem + 128;                                                   // [KV_BUFS][K rows | V rows]
    constexpr int BUFS = PUSH == 1 ? 1 : KV_BUFS;
    float *wt = reinterpret_cast<float *>(raw + BUFS * 2 * KV_HALF_BYTES);       // [8 heads][KV_WT_STRIDE]
    float *mw = wt + KV_MAX_GROUP * KV_WT_STRIDE;                                // [4 chunks, 4 pad][8 heads] maxima
    float *lw = mw + KV_MAX_GROUP * 8;                                           // ... and sums of the weights
    float *qd = lw + KV_MAX_GROUP * 8;                                           // [8 heads][8 blocks] query scales x `scale`
    uint32_t *q8 = reinterpret_cast<uint32_t *>(qd + KV_MAX_GROUP * 8);          // [8 heads][KV_Q_STRIDE]: 8 blocks x 8 words
    float *inbox = reinterpret_cast<float *>(q8 + KV_MAX_GROUP * KV_Q_STRIDE);   // PUSH: [CL ranks][GRP heads][dims of a slice], from every CTA of the cluster
    float2 *inbox_ml = reinterpret_cast<float2 *>(inbox + KV_MAX_GROUP * KV_D);  // PUSH: [CL ranks][8 heads] (m, l)

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int split = blockIdx.x, kvh = blockIdx.y;
    const int p_begin = split * chunk, p_end = min(p_begin + chunk, pos + 1);
    const int ntiles = p_end > p_begin ? (p_end - p_begin + KV_TILE - 1) / KV_TILE : 0;
    const uint8_t *kbase = K + (((size_t)layer * n_kv_head + kvh) * capacity) * KV_ROW;
    const uint8_t *vbase = V + (((size_t)layer * n_kv_head + kvh) * capacity) * KV_ROW;

    auto issue = [&](int i) {           // one thread
        const uint64_t pol = policy_evict_first();
        const int p0 = p_begin + i * KV_TILE, n = min(KV_TILE, p_end - p0), b = i % BUFS;
        const uint32_t bytes = (uint32_t)n * KV_ROW;
        uint8_t *dst = raw + (size_t)b * 2 * KV_HALF_BYTES;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_expect_tx(&kfull[b], bytes);
        bulk_g2s(dst, kbase + (size_t)p0 * KV_ROW, bytes, &kfull[b], pol);
        mbar_expect_tx(&vfull[b], bytes);
        bulk_g2s(dst + KV_HALF_BYTES, vbase + (size_t)p0 * KV_ROW, bytes, &vfull[b], pol);
    };
    float4 *halves = reinterpret_cast<float4 *>(inbox_ml + KV_WIDE_CLUSTER * KV_MAX_GROUP);      // PUSH: [8 warps][32] scores over half of the dims
    if (tid == 0) {
        for (int b = 0; b < BUFS; ++b) mbar_init(&kfull[b], 1), mbar_init(&vfull[b], 1);
        mbar_init(met, 1);
        mbar_fence_init();
        if (PUSH) mbar_expect_tx(met, CL * GRP * (KV_D / CL * 4 + 8));
    }
    for (int i = tid; i < KV_MAX_GROUP * KV_WT_STRIDE; i += THREADS) wt[i] = 0.0f;      // heads past the group stay 0
    for (int i = tid; i < KV_MAX_GROUP * 8; i += THREADS) qd[i] = 0.0f, mw[i] = 0.0f, lw[i] = 0.0f;
    for (int i = tid; i < KV_MAX_GROUP * KV_Q_STRIDE; i += THREADS) q8[i] = 0u;
    __syncthreads();
    if (PUSH) cluster_arrive();          // the others may write into this CTA's shared memory
    pdl_wait_prior_grid();              // q and the newest row of the cache come from the kernels before this one
    pdl_launch_dependents();
    if (tid == 0)
        for (int i = 0; i < min(ntiles, BUFS); ++i) issue(i);
    // the group's query heads, quantised as the cache rows are (host rule, src/kv_cache.h:100-117)
    {
        constexpr int ROUNDS = (GRP + WARPS - 1) / WARPS;
        const int blk = lane >> 2, sub = lane & 3;
        float x[ROUNDS][8], amax[ROUNDS];
#pragma unroll
        for (int r = 0; r < ROUNDS; ++r) {          // every load first: one trip to memory
            const int h = warp + r * WARPS;
            const float *qr = q + (size_t)(kvh * GRP + (h < GRP ? h : 0)) * KV_D + blk * 32 + sub * 8;
            if ((reinterpret_cast<uintptr_t>(q) & 15u) == 0) {
                const float4 a = *reinterpret_cast<const float4 *>(qr), c = *reinterpret_cast<const float4 *>(qr + 4);
                x[r][0] = a.x; x[r][1] = a.y; x[r][2] = a.z; x[r][3] = a.w; x[r][4] = c.x; x[r][5] = c.y; x[r][6] = c.z; x[r][7] = c.w;
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i) x[r][i] = qr[i];
            }
        }
#pragma unroll
        for (int r = 0; r < ROUNDS; ++r) amax[r] = kv_amax_8(x[r]);
        // the divisions of round r by lane r of the four
        static_assert(ROUNDS <= 4, "a lane of the four per round");
        float mine = amax[0];
#pragma unroll
        for (int r = 1; r < ROUNDS; ++r) mine = sub == r ? amax[r] : mine;
        const float d = __fdiv_rn(mine, 127.0f), my_id = d > 0.0f ? __fdiv_rn(1.0f, d) : 0.0f;
        if (warp + sub * WARPS < GRP && sub < ROUNDS) qd[(warp + sub * WARPS) * 8 + blk] = __fmul_rn(f16_bits_to_f32(f32_to_f16_bits_ties_away(d)), scale);
#pragma unroll
        for (int r = 0; r < ROUNDS; ++r) {
            const int h = warp + r * WARPS;
            const float id = __shfl_sync(0xffffffffu, my_id, (lane & ~3) + r);
            uint32_t w[2];
            kv_words_8(x[r], id, w);
            if (h < GRP) *reinterpret_cast<uint2 *>(q8 + h * KV_Q_STRIDE + blk * 8 + 2 * sub) = make_uint2(w[0], w[1]);
        }
    }
    __syncthreads();
    // B operand of the scores: head g, words t and t + 4 of every block, in the order the K rows are read in
    constexpr int QB = PUSH ? 4 : 8;                         // blocks of a warp
    uint32_t qb[QB][2];
#pragma unroll
    for (int b = 0; b < QB; ++b) {
        const uint32_t *src = q8 + g * KV_Q_STRIDE + (PUSH ? QB * (warp >> 2) + b : b) * 8;
        if (b & 1) {
            qb[b][0] = src[t];
            qb[b][1] = src[t + 4];
        } else {                        // even block: slot 0 = values 0, 1, 30, 31; slot i = values 4 i - 2 .. 4 i + 1
            qb[b][0] = t == 0 ? __byte_perm(src[0], src[7], 0x7610) : __byte_perm(src[t - 1], src[t], 0x5432);
            qb[b][1] = __byte_perm(src[t + 3], src[t + 4], 0x5432);
        }
    }
    const bool odd = NB == 1 && (warp & 1);                 // a warp of one block: whether it is the pair's second
    float m_run = -INFINITY, l_run = 0.0f;                  // of head g
    int top_run = 1;                                        // fp16 exponent of the largest V scale so far in the warp's two blocks
    float acc[NB][4][4];
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[b][j][i] = 0.0f;
    // The planes are of weight x scale x 2^(13 + 15 - top_run): the largest scale ends at 2^13 .. 2^14 (weights are at most 1), room for an
    // fp16 pair below.
    constexpr int LIFT = 127 + 13 + 15;

    for (int i = 0; i < (PUSH == 1 ? min(ntiles, 1) : ntiles); ++i) {
        const int b = i % BUFS;
        const uint32_t par = (uint32_t)((i / BUFS) & 1);
        const int n = min(KV_TILE, p_end - (p_begin + i * KV_TILE));
        uint8_t *kt = raw + (size_t)b * 2 * KV_HALF_BYTES, *vt = kt + KV_HALF_BYTES;
        bool ok = mbar_wait_hot(&kfull[b], par);
        {   // ---- scores of positions 16 (warp % 4) .. + 15; of eight warps over half of the dims each
            const int pw = warp & 3;
            const uint32_t *r0 = reinterpret_cast<const uint32_t *>(kt) + (size_t)(16 * pw + g) * (KV_ROW / 4);
            const uint32_t *r1 = r0 + 8 * (KV_ROW / 4);
            float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};          // (position g | g + 8, head 2 t | 2 t + 1), even blocks
            float so[4] = {0.0f, 0.0f, 0.0f, 0.0f};         // odd blocks: two short sums round less than a long one
#pragma unroll
            for (int i4 = 0; i4 < (PUSH ? 2 : 4); ++i4) {
                const int pr = PUSH ? 2 * (warp >> 2) + i4 : i4;
                const uint32_t *u0 = r0 + 17 * pr, *u1 = r1 + 17 * pr;
                const uint32_t d0 = u0[0], d1 = u1[0], e0 = u0[8], e1 = u1[8];
                uint32_t x0 = u0[t], x1 = u1[t];
                const uint32_t y0 = u0[t + 4], y1 = u1[t + 4];
                if (t == 0) {
                    x0 = __byte_perm(x0, e0, 0x5432);
                    x1 = __byte_perm(x1, e1, 0x5432);
                }
                int de[4], dq[4];
                mma_s8_16832(de, x0, x1, y0, y1, qb[2 * i4][0], qb[2 * i4][1]);
                mma_s8_16832(dq, u0[9 + t], u1[9 + t], u0[13 + t], u1[13 + t], qb[2 * i4 + 1][0], qb[2 * i4 + 1][1]);
                const float ke0 = half_bits_lo(d0), ke1 = half_bits_lo(d1), ko0 = half_bits_hi(e0), ko1 = half_bits_hi(e1);
                const float qe0 = qd[(2 * t) * 8 + 2 * pr], qe1 = qd[(2 * t + 1) * 8 + 2 * pr];
                const float qo0 = qd[(2 * t) * 8 + 2 * pr + 1], qo1 = qd[(2 * t + 1) * 8 + 2 * pr + 1];
                s[0] = __fmaf_rn(__fmul_rn(qe0, ke0), (float)de[0], s[0]);
                s[1] = __fmaf_rn(__fmul_rn(qe1, ke0), (float)de[1], s[1]);
                s[2] = __fmaf_rn(__fmul_rn(qe0, ke1), (float)de[2], s[2]);
                s[3] = __fmaf_rn(__fmul_rn(qe1, ke1), (float)de[3], s[3]);
                so[0] = __fmaf_rn(__fmul_rn(qo0, ko0), (float)dq[0], so[0]);
                so[1] = __fmaf_rn(__fmul_rn(qo1, ko0), (float)dq[1], so[1]);
                so[2] = __fmaf_rn(__fmul_rn(qo0, ko1), (float)dq[2], so[2]);
                so[3] = __fmaf_rn(__fmul_rn(qo1, ko1), (float)dq[3], so[3]);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) s[e] = __fadd_rn(s[e], so[e]);
            if (PUSH) {                              // the two warps of a group add their halves, both in the same order
                halves[warp * 32 + lane] = make_float4(s[0], s[1], s[2], s[3]);
                asm volatile("bar.sync %0, 64;" ::"r"(1 + pw) : "memory");
                const float4 a = halves[pw * 32 + lane], c = halves[(pw + 4) * 32 + lane];
                s[0] = __fadd_rn(a.x, c.x); s[1] = __fadd_rn(a.y, c.y); s[2] = __fadd_rn(a.z, c.z); s[3] = __fadd_rn(a.w, c.w);
            }
            const int pa = 16 * pw + g, pb = pa + 8;
            const bool va = pa < n, vb = pb < n;
            float mx0 = fmaxf(va ? s[0] : -INFINITY, vb ? s[2] : -INFINITY), mx1 = fmaxf(va ? s[1] : -INFINITY, vb ? s[3] : -INFINITY);
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) {
                mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, o));
                mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, o));
            }
            const float w0 = va ? expf(__fsub_rn(s[0], mx0)) : 0.0f, w1 = va ? expf(__fsub_rn(s[1], mx1)) : 0.0f;
            const float w2 = vb ? expf(__fsub_rn(s[2], mx0)) : 0.0f, w3 = vb ? expf(__fsub_rn(s[3], mx1)) : 0.0f;
            float l0 = __fadd_rn(w0, w2), l1 = __fadd_rn(w1, w3);
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) {
                l0 = __fadd_rn(l0, __shfl_xor_sync(0xffffffffu, l0, o));
                l1 = __fadd_rn(l1, __shfl_xor_sync(0xffffffffu, l1, o));
            }
            if (2 * t < GRP && warp < 4) {
                wt[(2 * t) * KV_WT_STRIDE + pa] = w0;
                wt[(2 * t) * KV_WT_STRIDE + pb] = w2;
                if (g == 0) mw[warp * 8 + 2 * t] = mx0, lw[warp * 8 + 2 * t] = l0;
            }
            if (2 * t + 1 < GRP && warp < 4) {
                wt[(2 * t + 1) * KV_WT_STRIDE + pa] = w1;
                wt[(2 * t + 1) * KV_WT_STRIDE + pb] = w3;
                if (g == 0) mw[warp * 8 + 2 * t + 1] = mx1, lw[warp * 8 + 2 * t + 1] = l1;
            }
        }
        ok = mbar_wait_hot(&vfull[b], par) && ok;
        if (n < KV_TILE)                // rows past the end: scales of zero (their weights are 0, but stale scales need not be finite)
            for (int z = tid; z < (KV_TILE - n) * 8; z += THREADS)
                reinterpret_cast<uint32_t *>(vt)[(n + (z >> 3)) * (KV_ROW / 4) + 17 * ((z >> 1) & 3) + 8 * (z & 1)] = 0u;
        // (the outcome of the bounded waits is made uniform: a CTA either goes on as a whole or leaves as a whole)
        if (!__syncthreads_and(ok ? 1 : 0)) break;
        {   // ---- values: dims 64 warp .. + 63, of eight warps 32 warp .. + 31
            const uint32_t *v32 = reinterpret_cast<const uint32_t *>(vt) + 17 * (NB == 2 ? warp : warp >> 1);
            uint32_t exps;                                  // which fp16 exponents the tile's scales have (0: none but zeros)
            {
                const uint32_t *ra = v32 + (size_t)lane * (KV_ROW / 4), *rb = ra + 32 * (KV_ROW / 4);
                auto exponent = [](uint32_t scale) { return min(scale, 1u) << (scale >> 10); };
                uint32_t mine = 0;
                if (NB == 2 || !odd) mine |= exponent(ra[0] & 0x7FFFu) | exponent(rb[0] & 0x7FFFu);
                if (NB == 2 || odd) mine |= exponent((ra[8] >> 16) & 0x7FFFu) | exponent((rb[8] >> 16) & 0x7FFFu);
                exps = __reduce_or_sync(0xffffffffu, mine);
            }
            float mc[4], m_new = m_run, f[4], lsum = 0.0f;
#pragma unroll
            for (int c = 0; c < 4; ++c) m_new = fmaxf(m_new, mc[c] = mw[c * 8 + g]);
            const float alpha = expf(__fsub_rn(m_run, m_new));
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                f[c] = expf(__fsub_rn(mc[c], m_new));
                lsum = __fmaf_rn(lw[c * 8 + g], f[c], lsum);
            }
            l_run = __fmaf_rn(l_run, alpha, lsum);
            m_run = m_new;
            const int top = max(top_run, 31 - __clz((int)(exps | 1u)));
            const bool wide = exps != 0u && top - ((exps & 1u) ? -9 : __ffs((int)exps) - 1) > KV_V_RANGE;      // warp-uniform
            const float up = __uint_as_float((uint32_t)(LIFT - top) << 23);
            const float keep = i == 0 ? 0.0f : __fmul_rn(alpha, __uint_as_float((uint32_t)(127 + top_run - top) << 23));      // a power of two: exact
            top_run = top;
            if (__any_sync(0xffffffffu, keep != 1.0f)) {
#pragma unroll
                for (int bb = 0; bb < NB; ++bb)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
#pragma unroll
                        for (int e = 0; e < 4; ++e) acc[bb][j][e] = __fmul_rn(acc[bb][j][e], keep);
            }
            // Two instructions' sums at a time: the tensor core cuts the last bits of a sum off, a rounded addition does not (all of
            // a split in one accumulator: relative error 3.2e-7 at 32768 positions, 2.6e-7 on the CUDA cores).
            auto weigh = [&](auto rest) {                   // rest: the second pass, over what the planes of the first left
                constexpr bool REST = decltype(rest)::value;
                float sum[NB][4][4];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    if (16 * c >= n) break;                     // CTA-uniform
                    if ((c & 1) == 0) {
#pragma unroll
                        for (int bb = 0; bb < NB; ++bb)
#pragma unroll
                            for (int j = 0; j < 4; ++j)
#pragma unroll
                                for (int e = 0; e < 4; ++e) sum[bb][j][e] = 0.0f;
                    }
                    const uint32_t *rows = v32 + (size_t)(16 * c + 2 * t) * (KV_ROW / 4);
                    uint32_t vals[NB][4];                       // four rows' bytes of a block, and their scales
                    float vd[NB][4];
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const uint32_t *u = rows + (size_t)((r & 1) + 8 * (r >> 1)) * (KV_ROW / 4);
                        const uint32_t d0 = u[0], e = u[8];
                        uint32_t x = NB == 1 && odd ? u[9 + g] : u[g];
                        if (g == 0 && !odd) x = __byte_perm(x, e, 0x5432);
                        vals[0][r] = x ^ 0x80808080u;
                        vd[0][r] = NB == 1 && odd ? half_bits_hi(e) : half_bits_lo(d0);
                        if constexpr (NB == 2) {
                            vals[1][r] = u[9 + g] ^ 0x80808080u;
                            vd[1][r] = half_bits_hi(e);
                        }
                    }
                    const float2 wa = *reinterpret_cast<const float2 *>(wt + g * KV_WT_STRIDE + 16 * c + 2 * t);
                    const float2 wb = *reinterpret_cast<const float2 *>(wt + g * KV_WT_STRIDE + 16 * c + 2 * t + 8);
                    const float fu = __fmul_rn(f[c], up);
#pragma unroll
                    for (int bb = 0; bb < NB; ++bb) {
                        const float *dd = vd[bb];
                        const uint32_t *vv = vals[bb];
                        uint32_t h01, l01, h23, l23;
                        const float p0 = __fmul_rn(__fmul_rn(wa.x, fu), dd[0]), p1 = __fmul_rn(__fmul_rn(wa.y, fu), dd[1]);
                        const float p2 = __fmul_rn(__fmul_rn(wb.x, fu), dd[2]), p3 = __fmul_rn(__fmul_rn(wb.y, fu), dd[3]);
                        split_f16x2(p0, p1, h01, l01);
                        split_f16x2(p2, p3, h23, l23);
                        if (REST) {
                            split_rest_f16x2(p0, p1, h01, l01);
                            split_rest_f16x2(p2, p3, h23, l23);
                        }
                        // byte j of four rows -> fp16: under the exponent of 1024 (value + 128, sign bit flipped above), minus 1152
                        const uint32_t p01 = __byte_perm(vv[0], vv[1], 0x5140), q01 = __byte_perm(vv[0], vv[1], 0x7362);
                        const uint32_t p23 = __byte_perm(vv[2], vv[3], 0x5140), q23 = __byte_perm(vv[2], vv[3], 0x7362);
                        const __half2 bias = __floats2half2_rn(1152.0f, 1152.0f);
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            uint32_t b0 = __byte_perm(j < 2 ? p01 : q01, 0x64646464u, (j & 1) ? 0x4342 : 0x4140);
                            uint32_t b1 = __byte_perm(j < 2 ? p23 : q23, 0x64646464u, (j & 1) ? 0x4342 : 0x4140);
                            const __half2 v0 = __hsub2(*reinterpret_cast<__half2 *>(&b0), bias), v1 = __hsub2(*reinterpret_cast<__half2 *>(&b1), bias);
                            mma_f16_16816(sum[bb][j], h01, l01, h23, l23, *reinterpret_cast<const uint32_t *>(&v0), *reinterpret_cast<const uint32_t *>(&v1));
                        }
                    }
                    if ((c & 1) == 1 || 16 * (c + 1) >= n) {
#pragma unroll
                        for (int bb = 0; bb < NB; ++bb)
#pragma unroll
                            for (int j = 0; j < 4; ++j)
#pragma unroll
                                for (int e = 0; e < 4; ++e) acc[bb][j][e] = REST ? __fmaf_rn(sum[bb][j][e], 0x1p-24f, acc[bb][j][e]) : __fadd_rn(acc[bb][j][e], sum[bb][j][e]);
                    }
                }
            };
            weigh(std::false_type{});
            if (__builtin_expect(wide, 0)) weigh(std::true_type{});
        }
        if (PUSH != 1) __syncthreads();                             // tile i's buffer and the tables may be overwritten
        if (PUSH != 1 && tid == 0 && i + BUFS < ntiles) issue(i + BUFS);
    }
    constexpr int SLICE = KV_D / CL;
    constexpr int OUTS = GRP * SLICE, ROUNDS = (OUTS + THREADS - 1) / THREADS;
    const float down = __uint_as_float((uint32_t)(254 - LIFT + top_run) << 23);
    auto part_of = [&](int bb, int j, int e) {                  // (of an infinity the low plane is NaN: the high plane alone is the sum then)
        const float high = acc[bb][j][e], both = isinf(high) ? high : __fadd_rn(high, acc[bb][j][e + 2]);
        return __fmul_rn(both, down);
    };
    if constexpr (PUSH) {
        // ---- every CTA's (m, l) goes to all of the cluster, its slices to the CTA that merges them, which counts the bytes: one trip, and nobody
        // reads another's memory
        cluster_wait();                                         // all have started
        const uint32_t me = cluster_rank();
        if (g < GRP) {
            float *box = inbox + ((int)me * GRP + g) * SLICE;
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int slot = 2 * t + e, dim = 32 * warp;
                if (odd) {
                    const int at = dim + 4 * slot;
                    st_async_f32x4(box + at % SLICE, met, (uint32_t)(at / SLICE), part_of(0, 0, e), part_of(0, 1, e), part_of(0, 2, e), part_of(0, 3, e));
                } else {
#pragma unroll
                    for (int j = 0; j < 4; j += 2) {            // the even block's values go in pairs: slot 0 has 0, 1 and 30, 31
                        const int at = dim + (slot == 0 ? (j == 0 ? 0 : 30) : 4 * slot - 2 + j);
                        st_async_f32x2(box + at % SLICE, met, (uint32_t)(at / SLICE), part_of(0, j, e), part_of(0, j + 1, e));
                    }
                }
            }
            if (warp < CL / 4) st_async_f32x2(reinterpret_cast<float *>(inbox_ml + me * KV_MAX_GROUP + g), met, (uint32_t)(4 * warp + t), m_run, l_run);
        }
        if (!__all_sync(0xffffffffu, mbar_wait_hot(met, 0))) {  // (nobody's bytes may find this CTA gone)
            cluster_arrive();
            cluster_wait();
            return;
        }
        if (tid / 32 * 32 >= OUTS) return;
        const int o = min(tid, OUTS - 1), h = o / SLICE, rr = lane & (CL - 1);
        static_assert(OUTS <= THREADS && (CL == SLICE || 32 % SLICE == 0) && CL <= SLICE, "lane rr of a head's CL weighs rank rr");
        float part[CL];
#pragma unroll
        for (int r = 0; r < CL; ++r) part[r] = inbox[r * OUTS + o];
        const float2 ml = inbox_ml[rr * KV_MAX_GROUP + h];
        float mx = ml.x;
#pragma unroll
        for (int i = 1; i < CL; i <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, i));
        const float w = ml.x == -INFINITY ? 0.0f : expf(__fsub_rn(ml.x, mx));          // a split without positions: 0
        float den = __fmul_rn(ml.y, w);
#pragma unroll
        for (int i = 1; i < CL; i <<= 1) den = __fadd_rn(den, __shfl_xor_sync(0xffffffffu, den, i));
        const float inv = __fdiv_rn(1.0f, den);
        float chain[CL / 4];                                    // of four ranks: sixteen in one sum round more than eight did
#pragma unroll
        for (int r = 0; r < CL; ++r) chain[r / 4] = __fmaf_rn(part[r], __shfl_sync(0xffffffffu, w, (lane & ~(CL - 1)) + r), r % 4 ? chain[r / 4] : 0.0f);
        float a = __fadd_rn(chain[0], chain[1]);
        if (CL == 16) a = __fadd_rn(a, __fadd_rn(chain[2], chain[CL / 4 - 1]));
        if (tid < OUTS) out[(size_t)kvh * GRP * KV_D + h * KV_D + (int)me * SLICE + o % SLICE] = __fmul_rn(a, inv);
        return;
    }
    // ---- the CTA's (m, l, acc); the tile buffers are free
    float *so = reinterpret_cast<float *>(raw), *sm = so + KV_MAX_GROUP * KV_D, *sl = sm + KV_MAX_GROUP;
    if (g < GRP) {
#pragma unroll
        for (int bb = 0; bb < NB; ++bb)
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int slot = 2 * t + e;
                    const int in_blk = bb ? 4 * slot + j : (slot == 0 ? (j < 2 ? j : 28 + j) : 4 * slot - 2 + j);
                    so[g * KV_D + 64 * warp + 32 * bb + in_blk] = part_of(bb, j, e);
                }
        if (warp == 0 && t == 0) sm[g] = m_run, sl[g] = l_run;
    }
    cluster_arrive();
    cluster_wait();
    // ---- one slice of the dims per CTA of the cluster, added over its CTAs in rank order
    const uint32_t rank = cluster_rank();
    const int n_cl = gridDim.x / CL, cl = blockIdx.x / CL;
    static_assert(PUSH || CL == KV_CLUSTER, "records and counters are laid out for clusters of eight");
    float *cw = wt, *cm = mw, *cl_sum = lw;                            // [8 heads][CL ranks] weights; maxima; denominators
    float part[ROUNDS][CL];
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        const int o = tid + r * KV_THREADS;
#pragma unroll
        for (int rr = 0; rr < CL; ++rr)
            part[r][rr] = o < OUTS ? ld_cluster_f32(so + (o / SLICE) * KV_D + (int)rank * SLICE + o % SLICE, (uint32_t)rr) : 0.0f;
    }
    static_assert(KV_MAX_GROUP * CL <= KV_THREADS, "a thread weighs one head of one rank");
    if (tid < KV_MAX_GROUP * CL) {
        const int h = tid / CL, rr = tid % CL;
        const float mm = h < GRP ? ld_cluster_f32(sm + h, (uint32_t)rr) : -INFINITY;
        const float ll = h < GRP ? ld_cluster_f32(sl + h, (uint32_t)rr) : 0.0f;
        float mx = mm;
#pragma unroll
        for (int o = 1; o < CL; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float w = mm == -INFINITY ? 0.0f : expf(__fsub_rn(mm, mx));      // a split without positions: 0
        float den = __fmul_rn(ll, w);
#pragma unroll
        for (int o = 1; o < CL; o <<= 1) den = __fadd_rn(den, __shfl_xor_sync(0xffffffffu, den, o));
        cw[h * CL + rr] = w;
        if (rr == 0) cm[h] = mx, cl_sum[h] = den;
    }
    __syncthreads();
    cluster_arrive();                   // this CTA has read its share of the others' memory (it leaves when all have: cluster_wait)
    float *rec = ws + (((size_t)kvh * CL + rank) * n_cl + cl) * KV_REC;
    float *out_slice = out + (size_t)kvh * GRP * KV_D + (int)rank * SLICE;
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        const int o = tid + r * KV_THREADS;
        if (o < OUTS) {
            const int h = o / SLICE;
            float chain[2] = {0.0f, 0.0f};      // of four ranks
#pragma unroll
            for (int rr = 0; rr < CL; ++rr) chain[rr / 4 % 2] = __fmaf_rn(part[r][rr], cw[h * CL + rr], chain[rr / 4 % 2]);
            const float a = __fadd_rn(chain[0], chain[1]);
            if (n_cl == 1) out_slice[h * KV_D + o % SLICE] = __fmul_rn(a, __fdiv_rn(1.0f, cl_sum[h]));
            else rec[o] = a;
        }
    }
    int last = 0;
    if (n_cl > 1) {
        if (tid < GRP) {
            rec[KV_MAX_GROUP * SLICE + tid] = cm[tid];
            rec[KV_MAX_GROUP * SLICE + KV_MAX_GROUP + tid] = cl_sum[tid];
        }
        __syncthreads();
        if (tid == 0) last = count_arrival(counters + kvh * CL + rank) == (unsigned int)n_cl - 1u;
        last = __syncthreads_or(last);
    }
    if (!last) {
        cluster_wait();
        return;
    }
    // ---- several clusters per head: the last one to bring this slice adds them in order (fixed, whichever is last).  All
    // loads go out before the weights are formed: one trip to L2 (a dependent trip per step took 5 us).
    if (tid == 0) counters[kvh * CL + rank] = 0u;
    const float *all = ws + ((size_t)kvh * CL + rank) * n_cl * KV_REC;
    constexpr int BATCH = 16, PAIRS = OUTS / 2;
    static_assert(PAIRS <= KV_THREADS, "a thread adds one pair of outputs");
    const int ho = min(tid, PAIRS - 1) / (SLICE / 2);
    float2 v[BATCH];
#pragma unroll
    for (int c = 0; c < BATCH; ++c)
        v[c] = (tid < PAIRS && c < n_cl) ? __ldcg(reinterpret_cast<const float2 *>(all + (size_t)c * KV_REC) + tid) : make_float2(0.0f, 0.0f);
    float *fm = reinterpret_cast<float *>(raw + 16384), *fl = fm + KV_MAX_CLUSTERS * KV_MAX_GROUP, *fw = fl + KV_MAX_CLUSTERS * KV_MAX_GROUP;
    for (int i = tid; i < n_cl * KV_MAX_GROUP; i += KV_THREADS) {
        const float *ml = all + (size_t)(i / KV_MAX_GROUP) * KV_REC + KV_MAX_GROUP * SLICE + i % KV_MAX_GROUP;
        const bool use = i % KV_MAX_GROUP < GRP;
        fm[i] = use ? __ldcg(ml) : 0.0f;
        fl[i] = use ? __ldcg(ml + KV_MAX_GROUP) : 0.0f;
    }
    __syncthreads();
    for (int i = tid; i < n_cl * KV_MAX_GROUP; i += KV_THREADS) {
        float mx = -INFINITY;
        for (int c = 0; c < n_cl; ++c) mx = fmaxf(mx, fm[c * KV_MAX_GROUP + i % KV_MAX_GROUP]);
        fw[i] = fm[i] == -INFINITY ? 0.0f : expf(__fsub_rn(fm[i], mx));
    }
    __syncthreads();
    if (tid < PAIRS) {
        float den = 0.0f, a = 0.0f, b = 0.0f;
        for (int c = 0; c < n_cl; ++c) den = __fmaf_rn(fl[c * KV_MAX_GROUP + ho], fw[c * KV_MAX_GROUP + ho], den);
#pragma unroll
        for (int c = 0; c < BATCH; ++c) {
            const float w = c < n_cl ? fw[c * KV_MAX_GROUP + ho] : 0.0f;
            a = __fmaf_rn(v[c].x, w, a);
            b = __fmaf_rn(v[c].y, w, b);
        }
        for (int c = BATCH; c < n_cl; ++c) {
            const float2 x = __ldcg(reinterpret_cast<const float2 *>(all + (size_t)c * KV_REC) + tid);
            a = __fmaf_rn(x.x, fw[c * KV_MAX_GROUP + ho], a);
            b = __fmaf_rn(x.y, fw[c * KV_MAX_GROUP + ho], b);
        }
        const float inv = __fdiv_rn(1.0f, den);
        float *o2 = out_slice + ho * KV_D + 2 * (tid % (SLICE / 2));
        o2[0] = __fmul_rn(a, inv);
        o2[1] = __fmul_rn(b, inv);
    }
    cluster_wait();
}

}  // namespace b200
