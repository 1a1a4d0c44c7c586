// ops.cuh -- the three entry points of the reference ABI that sit beside the mat-vec path: RMSNorm, the gated
// delta-net recurrent step and causal attention (include/bonsai_p40.h:44-56 in the reference).
//
// Oracles: src/ops.h:13-22 (rmsnorm), :66-92 (gdn_step) and the online-softmax recurrence of
// src/kernels/attn_p40.cu:92-118 / tests/test_p40.cpp:240-262.  The host code adds long sums sequentially and calls
// the C library's expf; the kernels add in a fixed tree order and use the device's expf, so outputs are held to
// 1e-5 of the largest output (the reference's own tests use 1e-4), not to the bit.
#pragma once

#include "activation.cuh"
#include "common.cuh"

namespace b200 {

// ---- sum of squares in the library's canonical order ------------------------------------------------------------
// A vector is cut into slices of 128 floats; inside a slice lane l adds x[4l]^2 .. x[4l+3]^2 in that order and a
// 5-step butterfly joins the lanes; slices are added in ascending order.  The fused producer of the list kernel
// (gemv_chain.cuh) uses the same order, so a fused RMSNorm gives the bits of this kernel.
__device__ __forceinline__ float lane_sumsq(float4 f) {
    float s = __fmul_rn(f.x, f.x);
    s = __fadd_rn(s, __fmul_rn(f.y, f.y));
    s = __fadd_rn(s, __fmul_rn(f.z, f.z));
    return __fadd_rn(s, __fmul_rn(f.w, f.w));
}
__device__ __forceinline__ float slice_sumsq(float4 f) {
    float s = lane_sumsq(f);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) s = __fadd_rn(s, __shfl_xor_sync(0xffffffffu, s, o));
    return s;
}
// 1 / sqrt(ss / n + eps), every step one IEEE operation (src/ops.h:13-17).
__device__ __forceinline__ float rms_scale(float ss, int n, float eps) {
    return __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, (float)n), eps)));
}
// silu(g) * u (src/ops.h:27-31); expf is the device's, not the host library's.
__device__ __forceinline__ float swiglu1(float g, float u) {
    return __fmul_rn(__fdiv_rn(g, __fadd_rn(1.0f, expf(-g))), u);
}

// VEC: four values per thread (n % 4 == 0, 16-byte aligned pointers).  EARLY: the next launch is let in at once, else by ending.
template <bool VEC, bool EARLY>
__global__ void __launch_bounds__(256) swiglu_kernel(const float *gate, const float *up, float *y, int n) {
    pdl_wait_prior_grid();
    if (EARLY) pdl_launch_dependents();
    const int i = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (VEC) {
        if (i < n / 4) {
            const float4 g = reinterpret_cast<const float4 *>(gate)[i], u = reinterpret_cast<const float4 *>(up)[i];
            reinterpret_cast<float4 *>(y)[i] = make_float4(swiglu1(g.x, u.x), swiglu1(g.y, u.y), swiglu1(g.z, u.z), swiglu1(g.w, u.w));
        }
    } else if (i < n) {
        y[i] = swiglu1(gate[i], up[i]);
    }
}

// One CTA per row.  VEC (n % 4 == 0, all pointers 16-byte aligned): 16-byte accesses; otherwise scalar ones, same order of
// sums.  HOLD > 0: rows of up to HOLD slices per warp stay in registers between the sum and the product, one trip to memory
// instead of two; HOLD <= 0 takes rows of any length; HOLD < 0 with few registers, for many CTAs per SM.  A row of less than
// eight slices has a warp per slice.  EARLY: as above.
constexpr int RMS_THREADS = 256, RMS_WARPS = RMS_THREADS / 32;
template <bool VEC>
__device__ __forceinline__ float4 rms_load(const float *p, int i, int n) {
    float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
    if (VEC) {
        if (i + 3 < n) f = *reinterpret_cast<const float4 *>(p + i);
    } else {
        if (i < n) f.x = p[i];
        if (i + 1 < n) f.y = p[i + 1];
        if (i + 2 < n) f.z = p[i + 2];
        if (i + 3 < n) f.w = p[i + 3];
    }
    return f;
}
template <bool VEC>
__device__ __forceinline__ void rms_store(float *p, int i, int n, float4 f, float sc, float4 w) {
    f.x = __fmul_rn(__fmul_rn(f.x, sc), w.x);
    f.y = __fmul_rn(__fmul_rn(f.y, sc), w.y);
    f.z = __fmul_rn(__fmul_rn(f.z, sc), w.z);
    f.w = __fmul_rn(__fmul_rn(f.w, sc), w.w);
    if (VEC) {
        if (i + 3 < n) *reinterpret_cast<float4 *>(p + i) = f;
    } else {
        if (i < n) p[i] = f.x;
        if (i + 1 < n) p[i + 1] = f.y;
        if (i + 2 < n) p[i + 2] = f.z;
        if (i + 3 < n) p[i + 3] = f.w;
    }
}
template <bool VEC, int HOLD, bool EARLY>
__global__ void __launch_bounds__(RMS_THREADS, HOLD < 0 || HOLD == 1 ? 8 : (HOLD == 8 && !VEC ? 3 : 0)) rmsnorm_kernel(const float *x, const float *w, float *y, int n, float eps) {
    constexpr int NW = RMS_WARPS;
    __shared__ __align__(16) float part[512];
    __shared__ float scale;
    const float *xr = x + (size_t)blockIdx.x * n;
    float *yr = y + (size_t)blockIdx.x * n;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int nslice = (n + 127) >> 7;
    pdl_wait_prior_grid();
    if (EARLY) pdl_launch_dependents();
    if constexpr (HOLD > 0) {
        float4 f[HOLD], g[HOLD];
#pragma unroll
        for (int r = 0; r < HOLD; ++r) f[r] = rms_load<VEC>(xr, (wid + NW * r) * 128 + 4 * lane, n);
#pragma unroll
        for (int r = 0; r < HOLD; ++r) g[r] = rms_load<VEC>(w, (wid + NW * r) * 128 + 4 * lane, n);
        // the slices' sums side by side (as slice_sumsq; past the end they are zeros), added by every warp for itself: one barrier (one after the other, and added
        // by one thread between two barriers: 8 rows of 5120 2.57 us, 2.18 now, 6144 2.84 and 2.47, 2048 rows of 5120 15.7 and 14.4).  Of one slice a warp one
        // thread still adds: many CTAs have no issue slots to spare (2048 rows of 1024 3.58, by every warp 4.08)
        float s[HOLD];
#pragma unroll
        for (int r = 0; r < HOLD; ++r) s[r] = lane_sumsq(f[r]);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
#pragma unroll
            for (int r = 0; r < HOLD; ++r) s[r] = __fadd_rn(s[r], __shfl_xor_sync(0xffffffffu, s[r], o));
#pragma unroll
        for (int r = 0; r < HOLD; ++r)
            if (lane == 0) part[wid + NW * r] = s[r];
        __syncthreads();
        float sc;
        if (HOLD > 1 || threadIdx.x == 0) {
            float acc = 0.0f;
#pragma unroll 2
            for (int k = 0; k + 4 <= nslice; k += 4) {
                const float4 p = *reinterpret_cast<const float4 *>(part + k);
                acc = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(acc, p.x), p.y), p.z), p.w);
            }
            for (int k = nslice & ~3; k < nslice; ++k) acc = __fadd_rn(acc, part[k]);
            sc = rms_scale(acc, n, eps);
            if (HOLD == 1) scale = sc;
        }
        if (HOLD == 1) {
            __syncthreads();
            sc = scale;
        }
#pragma unroll
        for (int r = 0; r < HOLD; ++r) rms_store<VEC>(yr, (wid + NW * r) * 128 + 4 * lane, n, f[r], sc, g[r]);
    } else {
        float acc = 0.0f;                           // rows longer than 512 slices: a part at a time, in ascending order
        for (int s0 = 0; s0 < nslice; s0 += 512) {
            for (int sl = s0 + wid; sl < min(nslice, s0 + 512); sl += NW) {
                const float s = slice_sumsq(rms_load<VEC>(xr, sl * 128 + 4 * lane, n));
                if (lane == 0) part[sl - s0] = s;
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                for (int k = 0; k < min(512, nslice - s0); ++k) acc = __fadd_rn(acc, part[k]);
                scale = rms_scale(acc, n, eps);
            }
            __syncthreads();
        }
        const float sc = scale;
        if (HOLD == 0) {
            for (int sl = wid; sl < nslice; sl += 4 * NW) {
                float4 f[4], g[4];
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    f[r] = rms_load<VEC>(xr, min(sl + NW * r, nslice) * 128 + 4 * lane, n);
                    g[r] = rms_load<VEC>(w, min(sl + NW * r, nslice) * 128 + 4 * lane, n);
                }
#pragma unroll
                for (int r = 0; r < 4; ++r) rms_store<VEC>(yr, min(sl + NW * r, nslice) * 128 + 4 * lane, n, f[r], sc, g[r]);
            }
        } else {
            const int nt = (int)blockDim.x;
            for (int i = threadIdx.x; i < n; i += 4 * nt) {          // (y may be x: the loads of a round first)
                float f[4], g[4];
#pragma unroll
                for (int r = 0; r < 4; ++r) f[r] = i + nt * r < n ? xr[i + nt * r] : 0.0f, g[r] = i + nt * r < n ? w[i + nt * r] : 0.0f;
#pragma unroll
                for (int r = 0; r < 4; ++r)
                    if (i + nt * r < n) yr[i + nt * r] = __fmul_rn(__fmul_rn(f[r], sc), g[r]);
            }
        }
    }
}

// ---- gated delta-net step ------------------------------------------------------------------------------------------
// state [n_v_heads][K][V]; one CTA per (value head, 32 state columns), 8 warps: lane = column, warp w holds rows
// w, w + 8, ... of the column in registers, so the state is read once and written once (2 * K * V * 4 bytes per head,
// the floor) and every access is a coalesced 128-byte row segment.  The column sums (k . S and q . S) are formed per
// warp over its rows in ascending order and joined across the warps in ascending warp order: a fixed order, not the
// host's strictly sequential one (src/ops.h:66-92) -- within the 1e-5 this operator is held to.  (A thread per whole
// column kept 128 values in registers and left 6144 threads for a 3 MB state: 45 us per call against 4 us for this shape.)
constexpr int GDN_KMAX = 128, GDN_WARPS = 8, GDN_RPW = GDN_KMAX / GDN_WARPS;
__global__ void __launch_bounds__(GDN_WARPS * 32) gdn_step_kernel(float *state, const float *q, const float *k, const float *v,
                                                                  const float *g, const float *beta, float *out, int n_k_heads, int n_v_heads, int K, int V) {
    __shared__ float ks[GDN_KMAX], qs[GDN_KMAX];
    __shared__ float part[GDN_WARPS][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tiles = V / 32;
    const int vh = blockIdx.x / tiles, vt = blockIdx.x - vh * tiles;
    const int j = vt * 32 + lane;
    const int kh = vh / (n_v_heads / n_k_heads);
    float *Sg = state + (size_t)vh * K * V + j;
    // the CTA's tile of the state, asked for while the launch before this one still runs: L2 hands out what it finds at the
    // load below, whoever writes in between
    // (and so are its row of v, its q and k, decay and step: behind the wait each was a trip to memory, 2.9 -> 2.6 us a step of 48, 3.0 -> 2.75 where a graph
    // replays them or their inputs are in memory)
    if ((int)threadIdx.x < K) {
        prefetch_l2(state + ((size_t)vh * K + threadIdx.x) * V + vt * 32);
    } else {
        const int i = 8 * ((int)threadIdx.x - K);
        if (i < K) prefetch_l2(k + (size_t)kh * K + i);
        else if (i < 2 * K) prefetch_l2(q + (size_t)kh * K + (i - K));
        else if (i < 2 * K + 32) prefetch_l2(v + (size_t)vh * V + vt * 32 + (i - 2 * K));
        else if (i < 2 * K + 40) prefetch_l2(g + vh);
        else if (i < 2 * K + 48) prefetch_l2(beta + vh);
    }
    pdl_wait_prior_grid();
    pdl_launch_dependents();
    float col[GDN_RPW];
#pragma unroll
    for (int r = 0; r < GDN_RPW; ++r) {
        const int i = warp + GDN_WARPS * r;
        col[r] = i < K ? Sg[(size_t)i * V] : 0.0f;
    }
    const float b = beta[vh], vj = v[(size_t)vh * V + j], decay = expf(g[vh]);
    for (int i = threadIdx.x; i < K; i += blockDim.x) {
        ks[i] = k[(size_t)kh * K + i];
        qs[i] = q[(size_t)kh * K + i];
    }
    __syncthreads();
    float kv = 0.0f;
#pragma unroll
    for (int r = 0; r < GDN_RPW; ++r) {
        const int i = warp + GDN_WARPS * r;
        if (i < K) {
            col[r] = __fmul_rn(col[r], decay);
            kv = __fadd_rn(kv, __fmul_rn(ks[i], col[r]));
        }
    }
    part[warp][lane] = kv;
    __syncthreads();
    kv = 0.0f;
#pragma unroll
    for (int w = 0; w < GDN_WARPS; ++w) kv = __fadd_rn(kv, part[w][lane]);
    __syncthreads();                                    // part is reused below
    const float d = __fsub_rn(vj, kv);
    float o = 0.0f;
#pragma unroll
    for (int r = 0; r < GDN_RPW; ++r) {
        const int i = warp + GDN_WARPS * r;
        if (i < K) {
            col[r] = __fadd_rn(col[r], __fmul_rn(__fmul_rn(b, ks[i]), d));
            o = __fadd_rn(o, __fmul_rn(qs[i], col[r]));
            Sg[(size_t)i * V] = col[r];
        }
    }
    part[warp][lane] = o;
    __syncthreads();
    if (warp == 0) {
        o = 0.0f;
#pragma unroll
        for (int w = 0; w < GDN_WARPS; ++w) o = __fadd_rn(o, part[w][lane]);
        out[(size_t)vh * V + j] = o;
    }
}

// ---- causal attention, head_dim 256 ------------------------------------------------------------------------------
// A warp owns FOUR consecutive queries of a head; lane l owns dimensions 8l .. 8l+7 of q and of the outputs.  The two or four
// warps of a CTA take 8 or 16 consecutive queries of ONE head (attn_redo: sixteen, 64), so they walk the same keys and values: a tile of 32 keys (K
// and V rows, 64 KB) is staged in shared memory once per CTA, and every row a warp reads from it serves four queries
// (with one query per warp the kernel was bound by shared-memory bandwidth: 2 KB read per (query, key)).  Scores: for
// eight keys at a time the lanes' partial dot products of the 4 x 8 (query, key) pairs go through one transposing
// reduction (31 shuffles for 32 scores instead of 5 per score), which leaves lane (query, key) with its score.  The
// softmax step is taken a tile at a time -- one running maximum, one rescale and four exps per lane per 32 keys: the
// online softmax of the reference's kernel (src/kernels/attn_p40.cu:101-113) with 32 keys per step instead of one.
// fp32 on the CUDA cores throughout; outputs are held to 1e-5 of the largest output.
constexpr int ATT_D = 256, ATT_TILE = 32, ATT_QPW = 4;
constexpr int att_smem_bytes(int warps) { return 2 * ATT_TILE * ATT_D * 4 + warps * ATT_TILE * ATT_QPW * 4; }

// part[r] of every lane -> returned value of lane r = sum over the lanes of part[r] (r = 0 .. 31).
__device__ __forceinline__ float transpose_sum32(float (&part)[32], int lane) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < o; ++i) {
            // the lane keeps the half of the values whose index has bit `o` equal to its own, and takes the partner's
            const float keep = up ? part[i + o] : part[i], give = up ? part[i] : part[i + o];
            part[i] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, give, o));
        }
    }
    return part[0];
}

// 16 bytes global -> shared, asynchronously, from L2 (whoever wrote them).
__device__ __forceinline__ void cp_async16(void *dst, const void *src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory"); }
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }

// Queries first .. first + 4 WARPS - 1 of one head, by a CTA of WARPS warps; smem: att_smem_bytes(WARPS), 16-byte aligned.  The next tile's keys are on
// their way while this one's values are multiplied, the next values while the next scores are.
template <int WARPS>
__device__ __forceinline__ void attn_simt(float *att_smem, const float *q, const float *k, const float *v, float *out, int first, int head,
                                          int n_tok, int n_head, int n_head_kv, float scale) {
    float (*kt)[ATT_D] = reinterpret_cast<float (*)[ATT_D]>(att_smem);
    float (*vt)[ATT_D] = reinterpret_cast<float (*)[ATT_D]>(att_smem + ATT_TILE * ATT_D);
    float4 *weights = reinterpret_cast<float4 *>(att_smem + 2 * ATT_TILE * ATT_D) + (threadIdx.x >> 5) * ATT_TILE;      // the warp's: [key of the tile][4 queries]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int q0 = first + ATT_QPW * warp;                  // the warp's first query
    const int kvh = head / (n_head / n_head_kv);
    const int myq = lane >> 3, mykk = lane & 7;             // after the reduction: lane = (query of the warp, key of the group of 8)
    float2 qreg[ATT_QPW][4], oreg[ATT_QPW][4];              // pairs of neighbouring dims
#pragma unroll
    for (int a = 0; a < ATT_QPW; ++a) {
        const int qi = q0 + a;
#pragma unroll
        for (int i = 0; i < 4; ++i) qreg[a][i] = oreg[a][i] = make_float2(0.0f, 0.0f);
        if (qi < n_tok) {
            const float *qp = q + ((size_t)qi * n_head + head) * ATT_D + 8 * lane;
#pragma unroll
            for (int i = 0; i < 4; ++i) qreg[a][i] = make_float2(__fmul_rn(qp[2 * i], scale), __fmul_rn(qp[2 * i + 1], scale));
        }
    }
    float m = -INFINITY, l = 0.0f;                          // of query q0 + myq (the same in the 8 lanes of its group)
    const int last = min(n_tok - 1, first + WARPS * ATT_QPW - 1);           // keys 0 .. last serve the CTA's queries
    const int wlast = min(n_tok - 1, q0 + ATT_QPW - 1);                     // ... 0 .. wlast this warp's
    auto stage = [&](float (*rows)[ATT_D], const float *from, int j0) {
        for (int i = threadIdx.x; i < min(ATT_TILE, last + 1 - j0) * (ATT_D / 4); i += WARPS * 32) {
            const int r = i / (ATT_D / 4), c4 = i % (ATT_D / 4);
            cp_async16(&rows[r][4 * c4], from + ((size_t)(j0 + r) * n_head_kv + kvh) * ATT_D + 4 * c4);
        }
        cp_async_commit();
    };
    stage(kt, k, 0);
    stage(vt, v, 0);
    for (int j0 = 0; j0 <= last; j0 += ATT_TILE) {
        const int nk = min(ATT_TILE, last + 1 - j0);
        const bool more = j0 + ATT_TILE <= last;            // CTA-uniform
        const bool live = q0 < n_tok && j0 <= wlast;        // warp-uniform: the warp's queries see keys of this tile
        cp_async_wait<1>();                                 // the keys
        __syncthreads();
        const int wn = live ? min(nk, wlast - j0 + 1) : 0;  // keys of this tile that any of the warp's queries may see
        float sc[4];
#pragma unroll
        for (int st = 0; st < 4; ++st) {
            sc[st] = -INFINITY;
            if (8 * st < wn) {                              // warp-uniform
                float part[32];
#pragma unroll
                for (int kk = 0; kk < 8; ++kk) {
                    const int r = 8 * st + kk;              // rows past wn hold stale data: masked below
                    const float4 ka = *reinterpret_cast<const float4 *>(&kt[r][8 * lane]);
                    const float4 kb = *reinterpret_cast<const float4 *>(&kt[r][8 * lane + 4]);
#pragma unroll
                    for (int a = 0; a < ATT_QPW; ++a) {
                        float2 pr = make_float2(__fmul_rn(qreg[a][0].x, ka.x), __fmul_rn(qreg[a][0].y, ka.y));
                        pr = fma2(qreg[a][1], make_float2(ka.z, ka.w), pr);
                        pr = fma2(qreg[a][2], make_float2(kb.x, kb.y), pr);
                        pr = fma2(qreg[a][3], make_float2(kb.z, kb.w), pr);
                        part[8 * a + kk] = __fadd_rn(pr.x, pr.y);
                    }
                }
                const float s = transpose_sum32(part, lane);            // lane (myq, mykk): score of key j0 + 8 st + mykk
                const int key = j0 + 8 * st + mykk;
                sc[st] = (key <= q0 + myq && key < n_tok && q0 + myq < n_tok) ? s : -INFINITY;
            }
        }
        __syncthreads();
        if (more) stage(kt, k, j0 + ATT_TILE);
        // softmax step of the tile, per query (groups of 8 lanes)
        float tmax = fmaxf(fmaxf(sc[0], sc[1]), fmaxf(sc[2], sc[3]));
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) tmax = fmaxf(tmax, __shfl_xor_sync(0xffffffffu, tmax, o));
        const float m_new = fmaxf(m, tmax);
        const float alpha = m_new == -INFINITY ? 1.0f : expf(__fsub_rn(m, m_new));      // a query with no key yet
        float p[4], psum = 0.0f;
#pragma unroll
        for (int st = 0; st < 4; ++st) {
            p[st] = sc[st] == -INFINITY ? 0.0f : expf(__fsub_rn(sc[st], m_new));
            psum = __fadd_rn(psum, p[st]);
            reinterpret_cast<float *>(weights)[(8 * st + mykk) * ATT_QPW + myq] = p[st];
        }
        if (more) cp_async_wait<1>();                       // the values
        else cp_async_wait<0>();
        __syncthreads();
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) psum = __fadd_rn(psum, __shfl_xor_sync(0xffffffffu, psum, o));
        l = __fadd_rn(__fmul_rn(l, alpha), psum);
        m = m_new;
#pragma unroll
        for (int a = 0; a < ATT_QPW; ++a) {
            const float al = __shfl_sync(0xffffffffu, alpha, 8 * a);
#pragma unroll
            for (int i = 0; i < 4; ++i) oreg[a][i] = make_float2(__fmul_rn(oreg[a][i].x, al), __fmul_rn(oreg[a][i].y, al));
        }
#pragma unroll 8
        for (int r = 0; r < wn; ++r) {                      // warp-uniform
            const float4 w4 = weights[r];
            const float w[ATT_QPW] = {w4.x, w4.y, w4.z, w4.w};
            const float4 va = *reinterpret_cast<const float4 *>(&vt[r][8 * lane]);
            const float4 vb = *reinterpret_cast<const float4 *>(&vt[r][8 * lane + 4]);
#pragma unroll
            for (int a = 0; a < ATT_QPW; ++a) {
                const float2 pp = make_float2(w[a], w[a]);
                oreg[a][0] = fma2(pp, make_float2(va.x, va.y), oreg[a][0]);
                oreg[a][1] = fma2(pp, make_float2(va.z, va.w), oreg[a][1]);
                oreg[a][2] = fma2(pp, make_float2(vb.x, vb.y), oreg[a][2]);
                oreg[a][3] = fma2(pp, make_float2(vb.z, vb.w), oreg[a][3]);
            }
        }
        __syncthreads();
        if (more) stage(vt, v, j0 + ATT_TILE);
    }
#pragma unroll
    for (int a = 0; a < ATT_QPW; ++a) {
        const int qi = q0 + a;
        const float la = __shfl_sync(0xffffffffu, l, 8 * a);
        if (qi < n_tok) {
            const float inv = __fdiv_rn(1.0f, la);
            float *op = out + ((size_t)qi * n_head + head) * ATT_D + 8 * lane;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                op[2 * i] = __fmul_rn(oreg[a][i].x, inv);
                op[2 * i + 1] = __fmul_rn(oreg[a][i].y, inv);
            }
        }
    }
}

// Bound by issue, and where the CTAs do not fill the SMs by a warp's chain: 8 us for a tile of 32 keys, five times its instructions, of which 1 - 2 were the
// wait for its rows (now copied asynchronously, a tile ahead).  Weights through shared memory instead of a shuffle for each of the lanes' 128, launches that
// begin while the one in front drains, CTAs of 16 or 8 queries (were 32): 24 heads over 4, us, before -> now: 1 token 4.7 -> 2.7, 16 8.3 -> 4.9, 30 12.1 -> 7.0, 70 18.5 ->
// 12.6, 100 26.7 -> 18.4, 130 34.7 -> 26.3, 191 49.2 -> 37.4; the same bits.  Shared memory holds three CTAs per SM of either size, and with the registers that three leave nothing is
// spilled (bound to four or eight, 128 registers a thread: 36 bytes; 100 tokens 19.6, 191 39.7; 64 heads 100 tokens 30.7, now 31.5, 191 62.1 and 60.8).
template <int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 3) attn_kernel(const float *q, const float *k, const float *v, float *out, int n_tok, int n_head, int n_head_kv, float scale) {
    extern __shared__ __align__(16) float att_smem[];
    // the longest rows of keys first: what starts last is short
    constexpr int QUERIES = WARPS * ATT_QPW;
    const int qblocks = (n_tok + QUERIES - 1) / QUERIES;
    const int head = (int)blockIdx.x % n_head, qb = qblocks - 1 - (int)blockIdx.x / n_head;
    pdl_wait_prior_grid();
    pdl_launch_dependents();
    attn_simt<WARPS>(att_smem, q, k, v, out, qb * QUERIES, head, n_tok, n_head, n_head_kv, scale);
}

}  // namespace b200
