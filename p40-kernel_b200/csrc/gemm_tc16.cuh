// gemm_tc16.cuh -- prefill mat-mul with the WHOLE contraction on the tensor cores (tcgen05.mma.kind::f16).
//
// gemm_tc.cuh keeps the integers of the host loop (one int8 MMA per 32-weight chunk, the per-chunk scales folded in
// by the CUDA cores) and is bound by exactly that fold.  This kernel moves the per-chunk activation scale to the OTHER side of the
// tensor core.  The dequantised activation  xh = da * a  (fp16 scale x int8, 18 significant bits) is split once per
// call into two fp16 numbers H + L = xh * 2^S exactly (S per token, a power of two that puts the token's largest
// value just under 2^15; L is the exact remainder, and where it underflows the loss is below 2^-38 of the token's
// largest value), the codes go to the tensor core as fp16 -1, 0, 1, 2, and one accumulator in tensor memory
// collects  sum_k (code_k - 1) * (H_k + L_k)  over a whole 128-weight block: products are exact, sums are the tensor
// core's fp32.  The CUDA cores are left with one fused multiply-add per output and BLOCK (the fp16 weight scale) and
// the expansion of the codes.
// Accuracy: the only roundings are the tensor core's fp32 additions inside a block (256 terms) and one fp32 FMA per
// block, against the host's one rounding per chunk term: Y is held to 1e-5 of max |Y| like the integer kernel's
// (measured ~1e-6); the INTEGERS of the host loop are not formed here: bonsai_b200_gemm_dump and
// bonsai_b200_set_option("gemm_path", 3) keep the integer kernel.
// Oracle: tests/test_p40.cpp:438-467 + src/pq2_0.h:149-169 (the host loop); kernel replaced: src/kernels/gemm_p40.cu:44-139.
//
// CTA tile 128 rows x 64 tokens, one CTA per SM, or 256 rows x 128 tokens by a pair of CTAs (cta_group::2: each has 128 rows of the
// codes in its tensor memory and 64 tokens' activations in its shared memory, and every MMA reads both CTAs' activations).  K is
// stepped one weight block at a time = 16 MMAs (M 128 per CTA, N the tile's tokens, K 16): two K halves of 64 values x {H, L} x four
// K = 16 steps, all into one accumulator (4 in flight at 64 tokens, 2 at 128).
//   epilogue   TN / 8 warps: per block two tcgen05.ld of 16 columns, acc += dw * D (one row x 32 tokens per thread)
//   producers  sets of four warps, thread = row: 128 two-bit codes -> 128 fp16, written to tensor memory; four sets in turn at 64 tokens,
//              each on a slot of its own, two at 128
//   issuers    two warps on alternate blocks, of a pair: the first CTA's
//   loaders    one warp each (tiled TMA copies): weight pieces of 8 blocks x 128 rows; a block's activations, two boxes of 64 values x
//              tokens x {H, L}, landing swizzled as the MMA reads them
// Block n of a CTA's walk lives in slot n % 4 of both rings.  One barrier per slot says that codes and activations are there (an arrival per
// producer warp, the loader's and its bytes), one that the block is multiplied: codes, activations and accumulator are handed
// on by the same commit.
#pragma once

#include "gemm_tc.cuh"

namespace b200 {

constexpr int T16_M = 128;                                 // weight rows of a CTA's tile
// The codes (A) never touch shared memory: the producers write the fp16 values straight into TENSOR memory (tcgen05.st, lane =
// weight row, 64 columns per block) and the MMA takes A from there -- with both operands in shared memory the tensor core's
// operand reads alone (6 KB per 128 x 64 x 16 MMA, 96 KB per block) ate 3/4 of the shared-memory bandwidth of the block's whole
// time budget.  The activations (B: the H and L planes of the tile's tokens) land in a shared-memory ring by TMA, asked for as far
// ahead as the ring allows: the boxes come from L2 and take ~1000-1500 cycles.
constexpr int T16_RING = 4;                                // blocks in flight: slots of the code ring and of the activation ring
constexpr int T16_A_COL0 = 256, T16_A_COLS = 64;           // tensor memory: accumulators in columns 0..255, then 4 blocks of codes x 64
constexpr int T16_SLOT_BYTES = 64 * 512;                   // activations of a block: 2 K halves x {H, L} x 64 tokens x 128 bytes
constexpr int T16_WBUFS = 2;
constexpr int T16_DWRING = 8;                              // weight scales of the last 8 blocks (the epilogue lags the producers)
constexpr int T16_ISSUERS = 2;                             // issuing warps: warp k takes the blocks n with n % 2 == k
constexpr int T16_TURN_STRIDE = 36, T16_TURN_FLOATS = 8 * T16_TURN_STRIDE;      // an epilogue warp turns 8 rows x 32 tokens round at once
constexpr int T16_PART_COUNTS = 16;                        // counts of a CTA whose share a tile begins in: one per epilogue warp
constexpr int T16_MAX_CTAS = 160;
// TN: the most tokens of a tile; CTAS: CTAs that multiply one tile together.
template <int TN, int CTAS>
struct T16C {
    static constexpr int ACC = 256 / TN;                                    // accumulators in flight (TN columns each)
    static constexpr int PART_FLOATS = T16_M * TN;                          // a CTA's slot for its part of a tile
    static constexpr int EPI_WARPS = TN / 8;                                // 4 lane quarters x (TN / 32) column groups of 32 tokens
    static constexpr int PROD_SETS = TN == 64 ? 4 : 2;                      // sets of producer warps, each on every fourth (second) block
    static constexpr int PROD_WARPS = 4 * PROD_SETS;                        // 4 row quarters per set
    static constexpr int THREADS = 32 * (EPI_WARPS + PROD_WARPS + T16_ISSUERS + 2);      // + weight loader, activation loader
    static constexpr int SMEM_BYTES = 2048 + T16_RING * T16_SLOT_BYTES + T16_DWRING * T16_M * 4 + T16_WBUFS * TC_WRAW_BYTES + EPI_WARPS * T16_TURN_FLOATS * 4;
    static_assert(TN / CTAS == 64, "a CTA's slot holds 64 tokens");
};
// Instruction descriptor: D = fp32, A and B fp16, both K-major; n tokens, 128 rows per CTA.
constexpr uint32_t t16_idesc(int n, int ctas) { return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(T16_M * ctas >> 4) << 24); }

struct T16Params {
    int n_out, nblocks, n_tok;
    int tile_n;                      // tokens of a tile: a multiple of 16 per CTA, at most TN
    int tiles_tok, n_tiles;          // token tiles per row tile, tiles in all (token tile runs fastest)
    int stream_k;                    // 1: contiguous ranges of (tile, block) iterations; 0: whole tiles, round-robin
    uint32_t idesc;
    long long per_worker;            // n_tiles * nblocks = per_worker * workers + rest
    int rest;
};

// The worker's (a CTA's or a pair's) next piece of work: blocks [kb0, kb1) of `tile`.  Every role walks the same sequence.
__device__ __forceinline__ long long t16_first(const T16Params &P, int worker, int workers) {
    return worker * P.per_worker + (long long)((uint32_t)(worker * P.rest) / (uint32_t)workers);
}
struct T16Walk {
    long long left;
    int tile, kb, step;
    __device__ __forceinline__ void start(const T16Params &P, int worker, int workers) {
        step = workers;
        if (P.stream_k) {
            const long long it = t16_first(P, worker, workers);
            left = t16_first(P, worker + 1, workers) - it;
            tile = it >> 32 ? (int)(it / P.nblocks) : (int)((uint32_t)it / (uint32_t)P.nblocks);
            kb = (int)(it - (long long)tile * P.nblocks);
        } else {
            tile = worker - workers;
            kb = 0;
        }
    }
    __device__ __forceinline__ bool next(const T16Params &P, int &t, int &kb0, int &kb1) {
        if (P.stream_k) {
            if (left <= 0) return false;
            t = tile++;
            kb0 = kb;
            kb1 = (int)min((long long)P.nblocks, kb + left);
            left -= kb1 - kb;
            kb = 0;
            return true;
        }
        tile += step;
        if (tile >= P.n_tiles) return false;
        t = tile;
        kb0 = 0;
        kb1 = P.nblocks;
        return true;
    }
};

// The descriptors' upper words are the same for every operand of this kernel (128-byte swizzle, 1024 bytes between
// 8-row groups); only the 14-bit address field of the lower word moves.  The issuing thread runs alone, one dependent
// instruction every few cycles, so an MMA is issued with two independent 32-bit adds and nothing else (building both
// 64-bit descriptors from an address cost ~75 cycles per MMA, 16 times per block).
constexpr uint32_t T16_DESC_HI = (uint32_t)(1024 >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint32_t tc16_desc_lo(uint32_t smem_addr) { return ((smem_addr >> 4) & 0x3FFFu) | (1u << 16); }
template <bool ACC, int CTAS = 1>
__device__ __forceinline__ void tc_mma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t idesc) {
    if (CTAS == 1)
        asm volatile(
            "{\n\t"
            ".reg .pred p;\n\t"
            ".reg .b64 db;\n\t"
            "mov.b64 db, {%2, %4};\n\t"
            "setp.ne.b32 p, %5, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %3, p;\n\t"
            "}\n"
            ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(idesc), "r"(T16_DESC_HI), "n"(ACC ? 1 : 0)
            : "memory");
    else
        asm volatile(
            "{\n\t"
            ".reg .pred p;\n\t"
            ".reg .b64 db;\n\t"
            "mov.b64 db, {%2, %4};\n\t"
            "setp.ne.b32 p, %5, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], db, %3, p;\n\t"
            "}\n"
            ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(idesc), "r"(T16_DESC_HI), "n"(ACC ? 1 : 0)
            : "memory");
}
// All of this thread's MMAs so far arrive on `bar`, of a pair: on both CTAs' barrier at this place.
template <int CTAS>
__device__ __forceinline__ void tc16_commit(uint32_t bar) {
    if (CTAS == 1)
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
    else
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3)
                     : "memory");
}
// The first CTA of the cluster's shared-memory address for this CTA's `addr`.
__device__ __forceinline__ uint32_t cluster_first(uint32_t addr) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
    return r;
}
// An arrival at a barrier of the pair's first CTA.  What it announces to the tensor core is ordered by the tcgen05 fence in front of it, so
// it needs no release at cluster scope (which costs 1200 cycles here: 2400 per block of 128 tokens instead of 1250).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Bounded wait in the unit's own blocking form (no time-out operand: with one the compiler makes a loop of a few dozen instructions
// of it), then as mbar_wait_bounded.  A barrier that has completed costs the waiting warp a third of mbar_wait_hot's instructions.
__device__ __forceinline__ bool mbar_wait_try(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        ".reg .u32 n;\n\t"
        "mov.u32 n, 4096;\n\t"
        "TRY_LOOP:\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "@p bra TRY_DONE;\n\t"
        "sub.u32 n, n, 1;\n\t"
        "setp.ne.u32 p, n, 0;\n\t"
        "@p bra TRY_LOOP;\n\t"
        "TRY_DONE:\n\t"
        "mov.u32 %0, n;\n\t"
        "}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0 || mbar_wait_bounded(bar, parity, 32, 128);
}
// Both of two barriers: their latencies lie beside each other.
__device__ __forceinline__ bool mbar_wait_both(uint64_t *bar0, uint32_t parity0, uint64_t *bar1, uint32_t parity1) {
    uint32_t ok;
    asm volatile(
        "{\n\t"
        ".reg .pred p, q;\n\t"
        ".reg .u32 n;\n\t"
        "mov.u32 n, 4096;\n\t"
        "BOTH_LOOP:\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 q, [%3], %4;\n\t"
        "and.pred p, p, q;\n\t"
        "@p bra BOTH_DONE;\n\t"
        "sub.u32 n, n, 1;\n\t"
        "setp.ne.u32 p, n, 0;\n\t"
        "@p bra BOTH_LOOP;\n\t"
        "BOTH_DONE:\n\t"
        "mov.u32 %0, n;\n\t"
        "}"
        : "=r"(ok)
        : "r"(smem_u32(bar0)), "r"(parity0), "r"(smem_u32(bar1)), "r"(parity1)
        : "memory");
    return ok != 0 || (mbar_wait_bounded(bar0, parity0, 32, 128) && mbar_wait_bounded(bar1, parity1, 32, 128));
}
__device__ __forceinline__ void tc_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};\n"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
          "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}
__device__ __forceinline__ void tc_st32(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};\n"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
          "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]),
          "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]),
          "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}
__device__ __forceinline__ void tc_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, int x, int y, int z, uint64_t *bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(smem_u32(dst)), "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
                 : "memory");
}
// The same for a CTA of a pair: the bytes are counted on `bar`, an address in the cluster's window.
__device__ __forceinline__ void tma_load_3d_pair(void *dst, const CUtensorMap *map, int x, int y, int z, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(smem_u32(dst)), "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ bool elect_one() {
    uint32_t pred;
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "}"
        : "=r"(pred));
    return pred != 0;
}
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int x, int y, uint64_t *bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(smem_u32(dst)), "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
                 : "memory");
}

// ---- once per call: the activations as two fp16 planes ------------------------------------------------------------
// 2^S for the token: S = 8 - exponent(max_c da_c), so that every |da * a * 2^S| < 2^15 (da = f * 2^ex, 0.5 <= f < 1,
// times 128 is below 2^(ex + 7)).
__device__ __forceinline__ int tc16_shift(unsigned int maxd_bits) {
    const float m = f16_bits_to_f32(maxd_bits);
    int ex = 0;
    if (m > 0.0f) (void)frexpf(m, &ex);
    return m > 0.0f ? 8 - ex : 0;
}
// Block = 4 tokens x one slice of the chunks (grid.y slices).  Every block first finds its tokens' largest chunk scale over
// ALL chunks -- a slice more reads the headers once more, from L2, and there is no pass, no zeroed array and no launch
// between the maximum and the split -- then thread = (chunk, token): 32 values -> 32 + 32 fp16, in the order the quantiser
// stored them (the order in which the code producers emit the codes).  planes: H at [tok][n_in], L at [n_tok + tok][n_in];
// scale[tok] = 2^-S for the epilogue.  A warp takes 4 tokens x 8 consecutive chunks: its stores are four runs of 512 bytes
// per plane.  Bound by launch and memory latency.  The first threads also clear the counts of the mat-mul's CTAs that share
// tiles, four at a time.
constexpr int T16_SPLIT_THREADS = 256, T16_SPLIT_PASS = T16_SPLIT_THREADS / 4;      // chunks of four tokens a block takes at once
template <bool FEW>
__global__ void __launch_bounds__(T16_SPLIT_THREADS) tc16_split_kernel(const uint32_t *Xq, int n_chunks, int n_tok, int slice, float *scale,
                                                                       __half *planes, uint4 *counts, int n_counts4) {
    __shared__ unsigned int top[T16_SPLIT_THREADS / 32][4];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tok = 4 * (int)blockIdx.x + (lane >> 3), c_first = (int)blockIdx.y * slice + 8 * warp + (lane & 7);
    pdl_wait_prior_grid();
    pdl_launch_dependents();
    // FEW blocks, about two per SM, wait for memory: the first own chunk flies beside the headers, and those four or eight at a time (indexes past
    // the end name the last one again).  With one trip after the other 37 tokens of 17408 took 6.5 us, 5.6 now, 512 of 5120 8.9 and 7.7.  With more
    // blocks the other way is ahead: 2048 tokens of 17408 65 us against 70.
    uint32_t w[9];
    auto fetch = [&](int c) {
        const uint32_t *src = Xq + 9 * ((size_t)min(c, n_chunks - 1) * n_tok + min(tok, n_tok - 1));
#pragma unroll
        for (int k = 0; k < 9; ++k) w[k] = src[k];
    };
    if (FEW) fetch(c_first);
    for (int i = ((int)blockIdx.y * (int)gridDim.x + (int)blockIdx.x) * T16_SPLIT_THREADS + (int)threadIdx.x; i < n_counts4;
         i += (int)(gridDim.x * gridDim.y) * T16_SPLIT_THREADS)
        counts[i] = make_uint4(0u, 0u, 0u, 0u);
    {   // four tokens are neighbours in memory: four lanes read one chunk's headers
        const int t = min(4 * (int)blockIdx.x + (lane & 3), n_tok - 1);
        unsigned int m = 0;
        int c = threadIdx.x >> 2;
        auto headers = [&](auto count) {
            constexpr int N = decltype(count)::value;
            unsigned int h[N];
#pragma unroll
            for (int k = 0; k < N; ++k) h[k] = Xq[9 * ((size_t)min(c + k * T16_SPLIT_PASS, n_chunks - 1) * n_tok + t)];
#pragma unroll
            for (int k = 0; k < N; ++k) m = max(m, h[k] & 0x7FFFu);
            c += N * T16_SPLIT_PASS;
        };
        if (FEW) {
            while (c + 4 * T16_SPLIT_PASS < n_chunks) headers(std::integral_constant<int, 8>());
            while (c < n_chunks) headers(std::integral_constant<int, 4>());
        } else {
#pragma unroll 4
            for (; c < n_chunks; c += T16_SPLIT_PASS) m = max(m, Xq[9 * ((size_t)c * n_tok + t)] & 0x7FFFu);
        }
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (lane < 4) top[warp][lane] = m;
    }
    __syncthreads();
    unsigned int m = 0;
#pragma unroll
    for (int k = 0; k < T16_SPLIT_THREADS / 32; ++k) m = max(m, top[k][lane >> 3]);
    if (tok >= n_tok) return;
    const int S = tc16_shift(m);
    const float up = ldexpf(1.0f, S);
    const size_t n_in = (size_t)n_chunks * 32;
    if (blockIdx.y == 0 && threadIdx.x < 32 && (lane & 7) == 0) scale[tok] = ldexpf(1.0f, -S);
    const int c1 = min(n_chunks, ((int)blockIdx.y + 1) * slice);
    for (int c = c_first; c < c1; c += T16_SPLIT_PASS) {
        if (!FEW || c != c_first) fetch(c);
        const float ds = __fmul_rn(f16_bits_to_f32(w[0] & 0xFFFFu), up);        // da * 2^S: exact (a power of two)
        uint4 *hp = reinterpret_cast<uint4 *>(planes + (size_t)tok * n_in + (size_t)c * 32);
        uint4 *lp = reinterpret_cast<uint4 *>(planes + ((size_t)n_tok + tok) * n_in + (size_t)c * 32);
        const int8_t *ab = reinterpret_cast<const int8_t *>(w + 1);      // the chunk's 32 int8 in stored order
#pragma unroll
        for (int q = 0; q < 4; ++q) {                       // 8 values per 16-byte store, in the order of tc16_expand
            uint32_t h[4], l[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                constexpr unsigned char PERM[16] = {0, 2, 4, 6, 8, 10, 12, 14, 1, 3, 5, 7, 9, 11, 13, 15};
                const int j0 = 16 * (q >> 1) + PERM[8 * (q & 1) + 2 * e], j1 = 16 * (q >> 1) + PERM[8 * (q & 1) + 2 * e + 1];
                const int a0 = (int)ab[j0], a1 = (int)ab[j1];
                const float v0 = __fmul_rn(ds, (float)a0), v1 = __fmul_rn(ds, (float)a1);      // exact: 11 x 7 bits
                const __half h0 = __float2half_rn(v0), h1 = __float2half_rn(v1);
                const __half l0 = __float2half_rn(__fsub_rn(v0, __half2float(h0))), l1 = __float2half_rn(__fsub_rn(v1, __half2float(h1)));
                h[e] = (uint32_t)__half_as_ushort(h0) | ((uint32_t)__half_as_ushort(h1) << 16);
                l[e] = (uint32_t)__half_as_ushort(l0) | ((uint32_t)__half_as_ushort(l1) << 16);
            }
            hp[q] = make_uint4(h[0], h[1], h[2], h[3]);
            lp[q] = make_uint4(l[0], l[1], l[2], l[3]);
        }
    }
}

// 16 two-bit codes of one word -> 16 fp16 (-1, 0, 1, 2) in eight words.  A code in bits p, p + 1 (p = 0, 2 .. 8) of a halfword that
// carries the exponent of 1024 is the fp16 number 1024 + 2^p code, so one three-input logic instruction makes two values and one
// packed multiply-add takes them to code - 1, exactly: 1024 2^-p + 1 has 11 bits.  9 instructions per word on the half-rate integer
// pipe, which this kernel kept busiest, and 8 on the multiply-add pipe (byte permutes whose selectors are the codes: 19 on the integer pipe).
// Order of the 16 values (the split kernel writes the activations in the same order): code (byte b, field k)
// of the word pairs with activation byte 4 k + b of the word's 16 (src/pq2_0.h:120-125, 158-166);
//   o[0..3] = (b0k0 b2k0) (b0k1 b2k1) (b0k2 b2k2) (b0k3 b2k3)   o[4..7]: the same for bytes 1 and 3.
template <int P>
__device__ __forceinline__ uint32_t tc16_pair(uint32_t w) {
    const uint32_t v = (w & (0x00030003u << P)) | 0x64006400u;
    const __half2 mul = __half2half2(__ushort_as_half((unsigned short)((15 - P) << 10)));               // 2^-P
    const __half2 sub = __half2half2(__float2half_rn(-(1024.0f / (float)(1 << P) + 1.0f)));
    const __half2 r = __hfma2(*reinterpret_cast<const __half2 *>(&v), mul, sub);
    return *reinterpret_cast<const uint32_t *>(&r);
}
__device__ __forceinline__ void tc16_expand(uint32_t w, uint32_t *o) {
    const uint32_t w8 = w >> 8;
    o[0] = tc16_pair<0>(w);
    o[1] = tc16_pair<2>(w);
    o[2] = tc16_pair<4>(w);
    o[3] = tc16_pair<6>(w);
    o[4] = tc16_pair<8>(w);
    o[5] = tc16_pair<2>(w8);
    o[6] = tc16_pair<4>(w8);
    o[7] = tc16_pair<6>(w8);
}
// acc += dw * v, each rounded once: two multiply-adds per instruction.
__device__ __forceinline__ void tc16_fold(float *acc, const int (&v)[16], float dw) {
#pragma unroll
    for (int i = 0; i < 16; i += 2)
        asm("{\n\t"
            ".reg .b64 x, y, z;\n\t"
            "mov.b64 x, {%2, %3};\n\t"
            "mov.b64 y, {%4, %4};\n\t"
            "mov.b64 z, {%0, %1};\n\t"
            "fma.rn.f32x2 z, x, y, z;\n\t"
            "mov.b64 {%0, %1}, z;\n\t"
            "}"
            : "+f"(acc[i]), "+f"(acc[i + 1]) : "r"(v[i]), "r"(v[i + 1]), "f"(dw));
}
// acc += dw0 * v0 + dw1 * v1, two of them per instruction: the two products are added first, so that a sum over n blocks is a chain of n / 2
// additions to a large number.
__device__ __forceinline__ void tc16_fold2(float *acc, const int (&v0)[8], float dw0, const int (&v1)[8], float dw1) {
#pragma unroll
    for (int i = 0; i < 8; i += 2)
        asm("{\n\t"
            ".reg .b64 x, y, z, t;\n\t"
            "mov.b64 x, {%2, %3};\n\t"
            "mov.b64 y, {%6, %6};\n\t"
            "mul.rn.f32x2 t, x, y;\n\t"
            "mov.b64 x, {%4, %5};\n\t"
            "mov.b64 y, {%7, %7};\n\t"
            "fma.rn.f32x2 t, x, y, t;\n\t"
            "mov.b64 z, {%0, %1};\n\t"
            "add.rn.f32x2 z, z, t;\n\t"
            "mov.b64 {%0, %1}, z;\n\t"
            "}"
            : "+f"(acc[i]), "+f"(acc[i + 1]) : "r"(v0[i]), "r"(v0[i + 1]), "r"(v1[i]), "r"(v1[i + 1]), "f"(dw0), "f"(dw1));
}
struct Tc16Maps {
    CUtensorMap w;        // PQ2_0 matrix as [n_out][row words], box 68 x 128
    CUtensorMap x;        // fp16 planes as [2][n_tok][n_in], box 64 values x a CTA's tokens of a tile x 2 planes, 128-byte swizzle
};

template <int TN, int CTAS>
__global__ void __launch_bounds__(T16C<TN, CTAS>::THREADS, 1) gemm_tc16_kernel(float *Y, const T16Params P, const float *tokscale,
                                                                               float *parts, unsigned int *counts, const __grid_constant__ Tc16Maps maps) {
    using C = T16C<TN, CTAS>;
    constexpr int EPI_WARPS = C::EPI_WARPS, PROD_WARPS = C::PROD_WARPS, SETS = C::PROD_SETS, ACC = C::ACC, COLS = 32;
    extern __shared__ __align__(128) uint8_t smem[];
    uint64_t *full = reinterpret_cast<uint64_t *>(smem);               // [4] producers and activation loader -> issuer (of a pair: the first CTA's is used)
    uint64_t *done = full + T16_RING;                                   // [4] tensor core -> producers, activation loader, epilogue
    uint64_t *acc_free = done + T16_RING;                               // [ACC] epilogue -> issuer (the first CTA's)
    uint64_t *wfull = acc_free + ACC;                                   // [2] weight loader -> producers
    uint64_t *wfree = wfull + T16_WBUFS;                                // [2] producers -> weight loader
    uint64_t *dwfull = wfree + T16_WBUFS;                               // [8] of a pair: producers -> epilogue, a block's scales are in the ring
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(dwfull + T16_DWRING);
    uint8_t *bring = smem + 1024 + ((1024u - (smem_u32(smem) & 1023u)) & 1023u);
    float *dwring = reinterpret_cast<float *>(bring + T16_RING * T16_SLOT_BYTES);
    uint8_t *wraw = reinterpret_cast<uint8_t *>(dwring + T16_DWRING * T16_M);
    float *turn = reinterpret_cast<float *>(wraw + T16_WBUFS * TC_WRAW_BYTES);

    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nblocks = P.nblocks, n_tok = P.n_tok, n_out = P.n_out;
    const int rank = CTAS == 1 ? 0 : (int)(blockIdx.x & 1), worker = (int)blockIdx.x / CTAS, workers = (int)gridDim.x / CTAS;
    const int epi_warps = min(EPI_WARPS, 4 * ((P.tile_n + COLS - 1) / COLS));        // those that have tokens
    constexpr int ISSUER = EPI_WARPS + PROD_WARPS, LOADER = ISSUER + T16_ISSUERS;
    T16Walk walk;
    walk.start(P, worker, workers);
    int tile, kb0, kb1;

    if (threadIdx.x == 0) {
        for (int s = 0; s < T16_RING; ++s) { mbar_init(&full[s], 4 * CTAS + 1); mbar_init(&done[s], 1); }
        for (int s = 0; s < ACC; ++s) mbar_init(&acc_free[s], CTAS * epi_warps);
        for (int s = 0; s < T16_DWRING; ++s) mbar_init(&dwfull[s], 4);
        mbar_fence_init();
    }
    if (threadIdx.x == LOADER * 32) {
        // the first piece of weights, which comes from memory, is asked for before anything else is set up
        for (int s = 0; s < T16_WBUFS; ++s) { mbar_init(&wfull[s], 1); mbar_init(&wfree[s], PROD_WARPS); }
        mbar_fence_init();
        T16Walk first = walk;
        if (first.next(P, tile, kb0, kb1)) {
            mbar_expect_tx(&wfull[0], (uint32_t)TC_WRAW_BYTES);
            tma_load_2d(wraw, &maps.w, (kb0 >> 3) * 68, (tile / P.tiles_tok) * (T16_M * CTAS) + T16_M * rank, &wfull[0]);
        }
        asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.x) : "memory");
    }
    if (wid == ISSUER) {
        if (CTAS == 1) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        }
    }
    tc_fence_before();
    if (CTAS == 1) __syncthreads();
    else asm volatile("barrier.cluster.arrive;\n\tbarrier.cluster.wait;" ::: "memory");
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (wid < EPI_WARPS) {
        // ---------------- epilogue: one weight row per thread, 32 tokens ----------------
        pdl_wait_prior_grid();                                           // token scales, counts and Y: the split's and its predecessors'
        const int q = wid & 3, cg = wid >> 2;
        const int row_l = 32 * q + lane;
        const bool second = COLS * cg + 16 < P.tile_n;
        const uint32_t tlane = tmem_base + ((uint32_t)(32 * q) << 16) + (uint32_t)(COLS * cg);
        const uint32_t acc_free0 = CTAS == 1 ? 0u : cluster_first(smem_u32(acc_free));
        bool ok = wid < epi_warps;
        int n = 0;
        while (ok && walk.next(P, tile, kb0, kb1)) {
            const int rt = tile / P.tiles_tok, tt = tile - rt * P.tiles_tok;
            const int row0 = rt * (T16_M * CTAS) + T16_M * rank + 32 * q, col0 = COLS * cg, tokb = tt * P.tile_n + col0;
            float acc[COLS];
#pragma unroll
            for (int j = 0; j < COLS; ++j) acc[j] = 0.0f;
            // At 64 tokens two blocks at a time (four accumulators): the waits of both lie beside each other, and the chain of rounded additions is
            // half as long (error against 64 bits 1.14e-7 -> 9.0e-8 at 5120, 1.44e-7 -> 1.13e-7 at 17408).
            for (int kb = kb0; kb < kb1; ++kb, ++n) {
                const int t = n & (ACC - 1);
                if (CTAS != 1 && !mbar_wait_try(&dwfull[n & (T16_DWRING - 1)], (uint32_t)((n / T16_DWRING) & 1))) { ok = false; break; }
                if (ACC == 4 && kb + 1 < kb1) {
                    const int n1 = n + 1, t1 = n1 & (ACC - 1);
                    if (!mbar_wait_both(&done[n & (T16_RING - 1)], (uint32_t)((n / T16_RING) & 1), &done[n1 & (T16_RING - 1)], (uint32_t)((n1 / T16_RING) & 1))) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const float dw = dwring[(n & (T16_DWRING - 1)) * T16_M + row_l], dw1 = dwring[(n1 & (T16_DWRING - 1)) * T16_M + row_l];
#pragma unroll
                    for (int h = 0; h < COLS; h += 8) {
                        if (h == 16 && !second) break;
                        int v[8], v1[8];
                        tc_ld8(tlane + (uint32_t)(t * TN + h), v);
                        tc_ld8(tlane + (uint32_t)(t1 * TN + h), v1);
                        tc_ld_wait();
                        tc16_fold2(acc + h, v, dw, v1, dw1);
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {                                     // the blocks' sums are in registers
                        mbar_arrive(&acc_free[t]);
                        mbar_arrive(&acc_free[t1]);
                    }
                    ++kb, ++n;
                    continue;
                }
                if (!mbar_wait_try(&done[n & (T16_RING - 1)], (uint32_t)((n / T16_RING) & 1))) { ok = false; break; }
                tc_fence_after();
                const float dw = dwring[(n & (T16_DWRING - 1)) * T16_M + row_l];
                if (CTAS == 1) {
#pragma unroll
                    for (int h = 0; h < COLS; h += 16) {
                        if (h == 16 && !second) break;
                        int v[16];
                        tc_ld16(tlane + (uint32_t)(t * TN + h), v);
                        tc_ld_wait();
                        tc16_fold(acc + h, v, dw);
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acc_free[t]);
                } else {
                    // Of a pair, whose two accumulators are what the tensor core waits for, all 32 columns are read before anything is done
                    // with them (256 tokens of 6144 -> 5120: 57.4 -> 56.4 us).
                    int v[16], v2[16];
                    tc_ld16(tlane + (uint32_t)(t * TN), v);
                    tc_ld16(tlane + (uint32_t)(t * TN + 16), v2);
                    tc_ld_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster(acc_free0 + 8u * (uint32_t)t);
                    tc16_fold(acc, v, dw);
                    tc16_fold(acc + 16, v2, dw);
                }
            }
            if (!ok) break;
            // ---- the tile (or this CTA's part of it) is done
            const int toks = min(min(COLS, P.tile_n - col0), n_tok - tokb);         // may be none
            const float scale = lane < toks ? tokscale[tokb + lane] : 0.0f;
            if (kb0 > 0 || kb1 < nblocks) {
                // A part of a tile that several workers share: left in this CTA's slot (one for the part at its start, one for the part at its end), four
                // tokens of a row per lane and store.  Whoever of a warp and its counterparts comes last adds the parts in the order of their blocks: nobody
                // waits for anybody, so the CTAs need not be resident at once and the launch need not be a cooperative one, which begins when everything
                // in front of it has ended.  (us, norm or SwiGLU and quantiser in front, cooperative with the first part's CTA waiting for the others / now: 37 tokens of 17408 ->
                // 5120 41.0 / 39.7, of 5120 -> 17408 32.3 / 28.6, 128 52.5 / 47.7, 64 of 1024 -> 5120 16.5 / 13.3, 20 of 5120 -> 5120 24.6 / 22.0, 512 of 5120 ->
                // 1024 41.4 / 41.1.  Letting the next launch start as soon as this one's wait is over costs 8 - 40 us where tiles are shared.)
                int head = worker, last = worker;
                const long long begin = (long long)tile * nblocks, end = begin + nblocks;
                while (t16_first(P, head, workers) > begin) --head;
                while (last + 1 < workers && t16_first(P, last + 1, workers) < end) ++last;
                auto slot_of = [&](int w) { return parts + ((size_t)(CTAS * w + rank) * 2 + (w == head ? 1 : 0)) * C::PART_FLOATS + (size_t)col0 * T16_M + row_l; };
                float *slot = slot_of(worker);
#pragma unroll
                for (int j0 = 0; j0 < COLS; j0 += 8) {
                    if (j0 >= toks) break;
#pragma unroll
                    for (int j = j0; j < j0 + 8; ++j) slot[j * T16_M] = acc[j];
                }
                __syncwarp();
                unsigned int before = 0;
                if (lane == 0) before = count_arrival(counts + (CTAS * head + rank) * T16_PART_COUNTS + wid);
                before = __shfl_sync(0xffffffffu, before, 0);
                if (before != (unsigned int)(last - head)) continue;
                __syncwarp();                               // what lane 0 acquired, every lane may read (a shuffle orders no memory)
                const float *from = slot_of(head);
#pragma unroll
                for (int j = 0; j < COLS; ++j) acc[j] = __ldcg(from + j * T16_M);
#pragma unroll 1
                for (int c = head + 1; c <= last; ++c) {
                    from = slot_of(c);
                    float t[COLS];
#pragma unroll
                    for (int j = 0; j < COLS; ++j) t[j] = __ldcg(from + j * T16_M);
#pragma unroll
                    for (int j = 0; j < COLS; ++j) acc[j] = __fadd_rn(acc[j], t[j]);
                }
            }
            // A row's tokens lie side by side in Y: turned round through shared memory eight rows at a time, a store writes 128 bytes of one
            // row.  (A row per lane, 16 bytes of 32 rows per store: 7000 cycles per tile of 128 tokens, in which both accumulators waited.)  The token's power-of-two scale is undone here.
            float *box = turn + wid * T16_TURN_FLOATS;
            float *y = Y + (size_t)row0 * n_tok + tokb + lane;
#pragma unroll 1
            for (int r0 = 0; r0 < 32; r0 += 8) {
                __syncwarp();
                if ((lane & 24) == r0) {
                    float4 *b = reinterpret_cast<float4 *>(box + (lane & 7) * T16_TURN_STRIDE);
#pragma unroll
                    for (int j = 0; j < COLS; j += 4) b[j / 4] = make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
                }
                __syncwarp();
                float v[8];
#pragma unroll
                for (int r = 0; r < 8; ++r) v[r] = box[r * T16_TURN_STRIDE + lane];
                if (lane < toks) {
                    // (a condition for all eight: one per row cost a hundred cycles each)
                    if (row0 + r0 + 8 <= n_out) {
#pragma unroll
                        for (int r = 0; r < 8; ++r) y[(size_t)r * n_tok] = __fmul_rn(v[r], scale);
                    } else {
#pragma unroll
                        for (int r = 0; r < 8; ++r)
                            if (row0 + r0 + r < n_out) y[(size_t)r * n_tok] = __fmul_rn(v[r], scale);
                    }
                }
                y += (size_t)8 * n_tok;
            }
        }
    } else if (wid < ISSUER) {
        // ---------------- code producers: thread = row, a set's every fourth (second) block ----------------
        // A warp reaches only the 32 tensor-memory lanes of its own quarter (warp index mod 4).  A warp takes both K halves of a block, one
        // after the other: its waits, addresses and arrivals are spent once per block (two sets of eight warps, a K half each: 5120 -> 17408
        // at 64 tokens 36.4 -> 35.0 us).
        const int pw = wid - EPI_WARPS, p = 32 * (pw & 3) + lane, set = pw >> 2;
        const uint32_t a_lane = tmem_base + ((uint32_t)(32 * (pw & 3)) << 16) + (uint32_t)T16_A_COL0;
        const uint32_t full0 = CTAS == 1 ? 0u : cluster_first(smem_u32(full));
        bool ok = true;
        int n = 0, oct = 0;
        while (ok && walk.next(P, tile, kb0, kb1)) {
            for (int kb = kb0; ok && kb < kb1; ++oct) {
                const int wbuf = oct % T16_WBUFS, end = min(kb1, (kb | 7) + 1);
                if (!mbar_wait_try(&wfull[wbuf], (uint32_t)((oct / T16_WBUFS) & 1))) { ok = false; break; }
                const uint8_t *rowp = wraw + (size_t)wbuf * TC_WRAW_BYTES + (size_t)p * 272;
                for (; kb < end; ++kb, ++n) {
                    if (SETS > 1 && (n & (SETS - 1)) != set) continue;
                    const int s = n & (T16_RING - 1);
                    // The block's eight code words sit at byte 34 j + 2 of the row's 272-byte piece, 2-byte aligned: nine aligned words and
                    // funnel shifts by 0 or 16 bits.  (Rows are 68 words apart: a warp's loads spread over eight banks, four passes each.)
                    const uint32_t off = (uint32_t)(kb & 7) * 34u + 2u;
                    const uint32_t *wa = reinterpret_cast<const uint32_t *>(rowp + (off & ~3u));
                    const uint32_t sh = (off & 2u) * 8u;
                    const uint32_t dbits = (uint32_t)*reinterpret_cast<const unsigned short *>(rowp + (kb & 7) * 34);
                    uint32_t x[9];
#pragma unroll
                    for (int i = 0; i < 9; ++i) x[i] = wa[i];
#pragma unroll
                    for (int g = 0; g < 2; ++g) {
                        uint32_t pc[32];
#pragma unroll
                        for (int i = 0; i < 4; ++i) tc16_expand(__funnelshift_r(x[4 * g + i], x[4 * g + i + 1], sh), pc + 8 * i);
                        if (g == 0) {
                            if (!mbar_wait_try(&done[s], (uint32_t)(((n / T16_RING) & 1) ^ 1))) { ok = false; break; }
                            tc_fence_after();
                        }
                        tc_st32(a_lane + (uint32_t)(s * T16_A_COLS + 32 * g), pc);     // 64 fp16 = 32 columns of this thread's lane
                    }
                    if (!ok) break;
                    dwring[(n & (T16_DWRING - 1)) * T16_M + p] = f16_bits_to_f32(dbits);
                    tc_st_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        if (CTAS == 1) mbar_arrive(&full[s]);
                        else mbar_arrive_cluster(full0 + 8u * (uint32_t)s);
                        if (CTAS != 1) mbar_arrive(&dwfull[n & (T16_DWRING - 1)]);
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&wfree[wbuf]);
            }
        }
    } else if (wid == LOADER) {
        // ---------------- weight loader: a piece (8 blocks x 128 rows, one tiled copy) as soon as its buffer is free ----------------
        int oct = 0;
        bool ok = true;
        while (ok && walk.next(P, tile, kb0, kb1)) {
            const int row = (tile / P.tiles_tok) * (T16_M * CTAS) + T16_M * rank;
            for (int kb = kb0; kb < kb1 && ok; kb = min(kb1, (kb | 7) + 1), ++oct) {
                const int wb = oct % T16_WBUFS;
                if (oct == 0) continue;                              // asked for at the start
                if (!mbar_wait_try(&wfree[wb], (uint32_t)(((oct / T16_WBUFS) & 1) ^ 1))) { ok = false; break; }
                if (elect_one()) {
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    mbar_expect_tx(&wfull[wb], (uint32_t)TC_WRAW_BYTES);
                    tma_load_2d(wraw + (size_t)wb * TC_WRAW_BYTES, &maps.w, (kb >> 3) * 68, row, &wfull[wb]);
                }
                __syncwarp();
            }
        }
    } else if (wid == LOADER + 1) {
        // ---------------- activation loader: a block's two boxes as soon as its slot is free ----------------
        pdl_wait_prior_grid();                                           // the planes
        const int bn = P.tile_n / CTAS;
        const uint32_t full0 = CTAS == 1 ? 0u : cluster_first(smem_u32(full));
        int n = 0;
        bool ok = true;
        while (ok && walk.next(P, tile, kb0, kb1)) {
            const int tok = (tile % P.tiles_tok) * P.tile_n + bn * rank;
            for (int kb = kb0; kb < kb1; ++kb, ++n) {
                const int s = n & (T16_RING - 1);
                if (!mbar_wait_try(&done[s], (uint32_t)(((n / T16_RING) & 1) ^ 1))) { ok = false; break; }
                if (elect_one()) {
                    uint8_t *b = bring + (size_t)s * T16_SLOT_BYTES;
                    if (rank == 0) mbar_expect_tx(&full[s], (uint32_t)(CTAS * bn * 512));          // both CTAs' bytes are counted on the first's barrier
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        if (CTAS == 1) tma_load_3d(b + h * bn * 256, &maps.x, kb * 128 + 64 * h, tok, 0, &full[s]);
                        else tma_load_3d_pair(b + h * bn * 256, &maps.x, kb * 128 + 64 * h, tok, 0, full0 + 8u * (uint32_t)s);
                    }
                }
                __syncwarp();
            }
        }
    } else if (rank == 0) {
        // ---------------- issuers: sixteen K = 16 MMAs per weight block, one accumulator ----------------
        // The whole warp walks the loop and waits; one elected lane issues.  Kept warp-uniform on purpose: the MMA takes
        // its operands from uniform registers, and inside a one-lane branch every operand had to be moved there first
        // (~70 cycles per MMA, measured).  A wait costs the warp 190 cycles even where its barrier has completed, and the queue behind it
        // holds a few MMAs only, so two warps take alternate blocks: one's waits lie beside the other's MMAs (alone with its waits and
        // commits, 16 MMAs of 64 tokens per block: 57 cycles each from one warp, 33 from two).  Blocks use different
        // accumulators, so their MMAs may interleave, and a commit covers the issuing thread's own MMAs.
        const uint32_t b_lo0 = tc16_desc_lo(smem_u32(bring)), half = (uint32_t)(P.tile_n / CTAS * 256) >> 4, plane = half >> 1;
        const uint32_t done0 = smem_u32(done), idesc = P.idesc;
        const int me = wid - ISSUER;
        bool ok = true;
        int n = 0;
        while (ok && walk.next(P, tile, kb0, kb1)) {
            const int skip = (n ^ me) & (T16_ISSUERS - 1);
            int m0 = n + skip;
            n += kb1 - kb0;
            for (int kb = kb0 + skip; kb < kb1; kb += T16_ISSUERS, m0 += T16_ISSUERS) {
                const int s = m0 & (T16_RING - 1), t = m0 & (ACC - 1);
                if (!mbar_wait_both(&full[s], (uint32_t)((m0 / T16_RING) & 1), &acc_free[t], (uint32_t)(((m0 / ACC) & 1) ^ 1))) { ok = false; break; }
                tc_fence_after();
                const uint32_t d = tmem_base + (uint32_t)(t * TN), a = tmem_base + (uint32_t)(T16_A_COL0 + s * T16_A_COLS);
                const uint32_t b = b_lo0 + (uint32_t)(s * (T16_SLOT_BYTES >> 4));
                if (elect_one()) {
#pragma unroll
                    for (int m = 0; m < 16; ++m) {
                        const uint32_t g = m >> 3, pl = (m >> 2) & 1, i = m & 3;              // K half, plane, K step: 16 fp16 = 8 columns of A
                        if (m == 0) tc_mma_f16_ts<false, CTAS>(d, a, b, idesc);
                        else tc_mma_f16_ts<true, CTAS>(d, a + 32u * g + 8u * i, b + g * half + pl * plane + 2u * i, idesc);
                    }
                    tc16_commit<CTAS>(done0 + 8u * (uint32_t)s);
                }
                __syncwarp();
            }
        }
    }
    tc_fence_before();
    // of a pair: neither CTA leaves while the other's MMAs or arrivals may still reach it
    if (CTAS == 1) __syncthreads();
    else asm volatile("barrier.cluster.arrive;\n\tbarrier.cluster.wait;" ::: "memory");
    if (wid == ISSUER) {
        tc_fence_after();
        if (CTAS == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

}  // namespace b200
