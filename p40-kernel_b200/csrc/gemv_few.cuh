// gemv_few.cuh -- one decode projection of few rows in ONE launch: y = W . Q8_1(FWHT(signs * x)).
//
// Same values as fwht_quant_kernel followed by gemv_stream_kernel, bit for bit: the same quantised blocks, the same terms
// (dw * da) * (float)sumi, added in the same order (gemv_stream.cuh: each of 8 lanes adds the terms of every 8th block of a
// segment in ascending order, a 3-step butterfly joins the lanes, segments are joined in ascending order).
//
// A projection of a thousand rows is a chain of latencies: 11 KB of weights per SM take less time than a launch.  So
//   * one launch instead of two (0.75 us between dependent launches on the device, 2 us on the host);
//   * the CTAs of a cluster rotate and quantise a share of the 1024-blocks each and send it to all of them (st.async: every
//     CTA counts the bytes that it gets);
//   * weights go from L2, where they are asked for in front of the wait, straight into registers while the rotation runs: a
//     warp's piece is (four rows) x (one step of 8 blocks), lane = (row, block), as in gemv_stream.cuh, but the steps of a
//     row are given to different warps, whose terms meet in shared memory to be added in order.  (One warp per four rows: 560
//     instructions in a chain behind the tables.)
//   * 10 warps of 70 registers (54 with one piece a warp): two CTAs per SM, so that the next launch's prologue runs beside this one.
// us per call, two launches -> this (in brackets: replayed by a graph): 5120 -> 64 4.54 -> 3.24 (3.78 -> 3.04), -> 1024 4.92 -> 3.91 (3.88 -> 3.68); 1024 ->
// 1024 4.16 -> 2.85 (3.33 -> 2.60); which calls take it and why: linear_one_launch.
#pragma once

#include "gemv_stream.cuh"

namespace b200 {

constexpr int FEW_WARPS = 10, FEW_HELD = 2, FEW_MAX_CLUSTER = 8;
inline int few_smem_bytes(int nb, int quads, int nseg) {
    return 16 + nb * (STREAM_ACT_WORDS + 4 + 4) * 4 + FWHT_N * 4 + quads * (nb / 8) * 32 * 16 + 4 * quads * nseg * 4;
}

// A cluster of nb / 8 CTAs (at most 8), each rotates the 1024-block of its rank; a CTA takes 4 * quads rows: quads * nb / 8 pieces, at most HELD per warp.
// seg_steps: steps of a segment (the last one takes what is left).
template <int HELD>
__global__ void __launch_bounds__(32 * FEW_WARPS, 2) gemv_few_kernel(const uint8_t *W, const float *x, const float *signs, float *y, uint32_t *xq_out,
                                                                     int n_out, int nb, int seg_steps, int quads) {
    extern __shared__ __align__(128) uint8_t smem[];
    uint64_t *tables = reinterpret_cast<uint64_t *>(smem);
    uint32_t *act_q = reinterpret_cast<uint32_t *>(smem + 16);
    float *act_s = reinterpret_cast<float *>(act_q + (size_t)nb * STREAM_ACT_WORDS);
    int *act_i = reinterpret_cast<int *>(act_s + (size_t)nb * 4);
    float4 *front = reinterpret_cast<float4 *>(act_i + (size_t)nb * 4);
    const int nfb = nb >> 3, mine = nfb == 1 ? 0 : (int)cluster_rank();
    float4 *terms = front + FWHT_N / 4;                 // [piece][lane]
    const int nseg = (nfb + seg_steps - 1) / seg_steps;
    float *sums = reinterpret_cast<float *>(terms + quads * nfb * 32);                  // [row][segment]

    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, rr = lane & 3, bl = lane >> 2;
    const int row0 = (int)blockIdx.x * 4 * quads, rows_here = min(4 * quads, n_out - row0);   // <= 0 in a CTA that fills up a cluster
    const size_t row_bytes = (size_t)nb * W_BLOCK_BYTES;
    if (nfb > 1) {
        if (threadIdx.x == 0) {
            mbar_init(tables, 1);
            mbar_fence_init();
            mbar_expect_tx(tables, (uint32_t)nb * 4 * (32 + 4 + 4));
        }
        __syncwarp();
        cluster_arrive();                               // this CTA runs: the others may store into its tables
    }
    // (whoever wrote them, a request to bring them into L2 is harmless)
    if (threadIdx.x == 32) {
        if (rows_here > 0) bulk_prefetch_l2(W + (size_t)row0 * row_bytes, (uint32_t)(rows_here * row_bytes));
        bulk_prefetch_l2(x + (size_t)mine * FWHT_N, FWHT_N * 4);
        if (signs) bulk_prefetch_l2(signs + (size_t)mine * FWHT_N, FWHT_N * 4);
    }
    pdl_wait_prior_grid();
    pdl_launch_dependents();

    const bool rotates = wid < 8;                       // a warp per slice of 128
    const size_t at = (size_t)mine * FWHT_N + wid * 128 + 4 * lane;
    float4 f = make_float4(1.f, 1.f, 1.f, 1.f), sg = f;
    if (rotates) {
        f = *reinterpret_cast<const float4 *>(x + at);
        if (signs) sg = *reinterpret_cast<const float4 *>(signs + at);
    }
    // the weights: rows past the end name the last one again, their sums are not stored
    const int pieces = rows_here > 0 ? quads * nfb : 0;
    uint32_t w[HELD][9];
    float dw[HELD];
#pragma unroll
    for (int k = 0; k < HELD; ++k) {
        const int u = min(wid + FEW_WARPS * k, quads * nfb - 1), quad = u / nfb, b = bl + 8 * (u - quad * nfb);
        const uint8_t *blk = W + (size_t)min(row0 + 4 * quad + rr, n_out - 1) * row_bytes + (size_t)W_BLOCK_BYTES * b;
        const uint32_t *p = reinterpret_cast<const uint32_t *>(blk + ((b & 1) ? 2 : 0));     // an even block starts on a word, an odd one's codes do
#pragma unroll
        for (int i = 0; i < 8; ++i) w[k][i] = p[i];
        w[k][8] = (b & 1) ? 0u : (uint32_t)*reinterpret_cast<const unsigned short *>(blk + 32);
        dw[k] = f16_bits_to_f32((b & 1) ? (uint32_t)*reinterpret_cast<const unsigned short *>(blk) : w[k][0] & 0xFFFFu);
    }
    if (nfb > 1) cluster_wait();                         // all have started
    if (rotates) {
        float v[4] = {f.x, f.y, f.z, f.w};
        if (signs) {
            v[0] = __fmul_rn(v[0], sg.x); v[1] = __fmul_rn(v[1], sg.y);
            v[2] = __fmul_rn(v[2], sg.z); v[3] = __fmul_rn(v[3], sg.w);
        }
        fwht_slice_front(v, lane);
        front[wid * 32 + lane] = make_float4(v[0], v[1], v[2], v[3]);
    }
    __syncthreads();
    if (rotates) {
        float v[4];
        uint32_t word, header;
        fwht_slice_back(front, wid, lane, v);
        quantise_chunk_8lanes(v, lane, word, header);
        const int chunk = 32 * mine + 4 * wid + (lane >> 3);
        if (nfb == 1) put_activation<1>(act_q, act_s, act_i, tables, chunk, lane, word, header);
        else put_activation<0>(act_q, act_s, act_i, tables, chunk, lane, word, header, nfb);
        if ((int)blockIdx.x < nfb) {                    // the first cluster leaves the blocks where the two launches would have
            xq_out[9 * chunk + 1 + (lane & 7)] = word;
            if ((lane & 7) == 0) xq_out[9 * chunk] = header;
        }
    }
    bool ok = true;
    if (nfb == 1) __syncthreads();
    else ok = mbar_wait_hot(tables, 0);
#pragma unroll
    for (int k = 0; k < HELD; ++k) {
        const int u = wid + FEW_WARPS * k;
        if (u >= pieces) break;                         // warp-uniform
        const int b = bl + 8 * (u % nfb);
        const uint32_t sh = (b & 1) ? 0u : 16u;
        const float4 sc = *reinterpret_cast<const float4 *>(act_s + 4 * b);
        const int4 in = *reinterpret_cast<const int4 *>(act_i + 4 * b);
        const float scale[4] = {sc.x, sc.y, sc.z, sc.w};
        const int inits[4] = {in.x, in.y, in.z, in.w};
        float t[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int4 lo = *reinterpret_cast<const int4 *>(act_q + b * STREAM_ACT_WORDS + c * 8);
            const int4 hi = *reinterpret_cast<const int4 *>(act_q + b * STREAM_ACT_WORDS + c * 8 + 4);
            const int a[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
            const uint32_t c0 = __funnelshift_r(w[k][2 * c], w[k][2 * c + 1], sh);
            const uint32_t c1 = __funnelshift_r(w[k][2 * c + 1], w[k][2 * c + 2], sh);
            t[c] = __fmul_rn(__fmul_rn(dw[k], scale[c]), (float)chunk_sumi_scaled(c0, c1, a, inits[c]));
        }
        terms[u * 32 + lane] = make_float4(t[0], t[1], t[2], t[3]);
    }
    // (a warp whose wait ran out comes here too, with terms of whatever lies in the tables: the CTA leaves as a whole)
    if (!__syncthreads_and(ok ? 1 : 0)) {
        if (nfb > 1) {                                  // nobody's bytes may find this CTA gone
            cluster_arrive();
            cluster_wait();
        }
        return;
    }
    for (int i = wid; i < (pieces ? quads * nseg : 0); i += FEW_WARPS) {
        const int quad = i / nseg, j = i - quad * nseg;
        float acc = 0.0f;
        for (int s = j * seg_steps; s < min(nfb, (j + 1) * seg_steps); ++s) {
            const float4 t = terms[(quad * nfb + s) * 32 + lane];
            acc = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(acc, t.x), t.y), t.z), t.w);
        }
        acc = __fadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, 4));
        acc = __fadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, 8));
        acc = __fadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, 16));
        if (nseg > 1) {
            if (bl == 0) sums[(4 * quad + rr) * nseg + j] = acc;
        } else if (bl == 0 && 4 * quad + rr < rows_here) {
            y[row0 + 4 * quad + rr] = acc;
        }
    }
    if (nseg > 1) {
        __syncthreads();
        if ((int)threadIdx.x < rows_here) {
            float total = sums[threadIdx.x * nseg];
            for (int j = 1; j < nseg; ++j) total = __fadd_rn(total, sums[threadIdx.x * nseg + j]);
            y[row0 + threadIdx.x] = total;
        }
    }
}

}  // namespace b200
