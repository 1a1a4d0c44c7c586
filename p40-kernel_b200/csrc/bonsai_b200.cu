// bonsai_b200.cu -- the C-ABI of the sm_100a build: argument checks, launch geometry, launches.
//
// One translation unit on purpose: every kernel shares the device status word of common.cuh.
// Host side mirrors the reference wrappers (src/kernels/gemv_p40.cu:200-219, gemm_p40.cu:143-154,
// gemv_repack_p40.cu:196-220, elementwise_p40.cu:75-80): validate, compute a grid, launch on the
// caller's stream, return cudaGetLastError().  No allocation, no synchronisation, no CPU fallback.
#include "../../include/bonsai_b200_ext.h"
#include "../../include/bonsai_kv.h"

#include "activation.cuh"
#include "attn_tc.cuh"
#include "gemm_simt.cuh"
#include "gemm_tc.cuh"
#include "gemm_tc16.cuh"
#include "gemv.cuh"
#include "gemv_stream.cuh"
#include "gemv_chain.cuh"
#include "gemv_few.cuh"
#include "gemv_mma.cuh"
#include "kv.cuh"
#include "ops.cuh"
#include "probe.cuh"
#include "ptq.cuh"
#include "repack.cuh"
#include "scratch.cuh"
#include "synth.cuh"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <iterator>
#include <mutex>
#include <new>
#include <type_traits>
#include <utility>
#include <vector>

using namespace b200;

namespace {

constexpr int SM_COUNT = 148;                 // B200
constexpr int SMEM_LIMIT = 227 * 1024;        // dynamic shared memory a CTA may opt into

std::atomic<int> g_opt_pdl{0};
std::atomic<int> g_opt_overlap{1};             // 0: plain launches, each begins when its predecessor has ended
std::atomic<int> g_opt_gemv_variant{-1};
std::atomic<int> g_opt_gemv_order{0};
std::atomic<int> g_opt_fuse_linear{-1};        // bonsai_b200_linear: -1 one kernel or two by shape, 0 two, 1 one when it can
std::atomic<int> g_opt_chain_threads{512};       // threads per CTA of the chain kernel: 512 (5 blocks per lane and task), 640 (4), 768 (3)
// Dependent ops with at least this many blocks per row rotate their input once for the grid instead of once per CTA; 0 = never.  us per op of a list
// n -> n, once per CTA / once for the grid: 1024 behind a norm 5.2 / 5.7, 2048 6.4 / 6.2 (plain 5.5 / 5.35), 3072 7.3 / 6.8, 5120 9.6 / 8.1.
std::atomic<int> g_opt_chain_spread_nb{16};
std::atomic<int> g_opt_chain_tile_kb{16};
std::atomic<int> g_opt_kv_wide{1};                // decode attention: 0 = clusters of eight CTAs at every length
std::atomic<int> g_opt_kv_push{1};                // ... 0 = of the eight the form for several clusters at every length
std::atomic<int> g_opt_gemm_tile{0};              // fp16 tensor-core mat-mul: 0 by estimated time, else tiles of up to 64 tokens (a CTA) or 128 (a pair)
std::atomic<int> g_opt_chain_seg{40};            // longest row segment of one task, in blocks: 8, 16, 24, 32 or 40        // target bytes of one ring slot
std::atomic<int> g_opt_gemm_path{-1};          // -1: by token count, 0: integer SIMT kernel, 1: tensor cores, 2: small-batch kernel, 3: integer tensor-core kernel          // 0: streaming kernel (fixed tree order), 1: the host's sequential order

inline cudaStream_t as_stream(bonsai_stream s) { return reinterpret_cast<cudaStream_t>(s); }
inline bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
inline bool aligned4(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 3u) == 0; }

// cudaFuncSetAttribute is per device; remember which devices have been configured per kernel.
struct SmemOptIn {
    std::atomic<unsigned long long> done{0};
    template <typename K>
    cudaError_t ensure(K kernel) {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        const unsigned long long bit = 1ull << (dev & 63);
        if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT);
        if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
        return e;
    }
};

template <typename... KArgs, typename... Args>
cudaError_t launch(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, bool pdl,
                   Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    if (pdl && g_opt_overlap.load()) {
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// Launches in clusters of CTAs, which a device, a limit on its SMs or a tool may refuse (a profiler that replays kernels: cooperative ones).
std::atomic<int> g_opt_refuse_clusters{0};        // test build: so many of them are refused without being tried
template <typename... KArgs, typename... Args>
cudaError_t launch_clusters(const cudaLaunchConfig_t &cfg, void (*kernel)(KArgs...), Args... args) {
    if (g_opt_refuse_clusters.load() > 0 && g_opt_refuse_clusters.fetch_sub(1) > 0) return cudaErrorInvalidConfiguration;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}
// Clusters of a kernel that are resident at once with an SM for each CTA, per device: asked once; none from the first launch on that was refused.
class ClusterRoom {
public:
    template <typename K>
    int ask(K kernel, SmemOptIn &opt, unsigned cluster, unsigned threads) {
        int dev = 0, resident = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || dev >= 64) return 0;
        if ((resident = known_[dev].load(std::memory_order_relaxed)) != 0) return std::max(resident, 0);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(SM_COUNT / cluster * cluster);
        cfg.blockDim = dim3(threads);
        cfg.dynamicSmemBytes = SMEM_LIMIT;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = cluster;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if (opt.ensure(kernel) != cudaSuccess || cudaOccupancyMaxActiveClusters(&resident, kernel, &cfg) != cudaSuccess || resident <= 0) {
            (void)cudaGetLastError();
            resident = -1;
        }
        known_[dev].store(resident, std::memory_order_relaxed);
        return std::max(resident, 0);
    }
    // Whether e says that clusters are not launched here; no later call tries them then.
    bool refused(cudaError_t e) {
        if (e != cudaErrorInvalidConfiguration && e != cudaErrorCooperativeLaunchTooLarge && e != cudaErrorNotSupported) return false;
        (void)cudaGetLastError();
        int dev = 0;
        if (cudaGetDevice(&dev) == cudaSuccess && dev < 64) known_[dev].store(-1, std::memory_order_relaxed);
        return true;
    }
#ifdef BONSAI_B200_TUNING
    void forget() {
        for (auto &k : known_) k.store(0, std::memory_order_relaxed);
    }
#endif

private:
    std::atomic<int> known_[64] = {};
};

ClusterRoom g_tc16_pairs, g_repack_pairs, g_repack_fours, g_few_clusters[FEW_MAX_CLUSTER + 1];
SmemOptIn g_few_opt[FEW_HELD];

// ceil(2^32 / d): __umulhi(n, magic) == n / d for every n with n * d < 2^32; 0 stands for d == 1.
inline uint32_t magic_u32(uint32_t d) {
    if (d <= 1) return 0u;
    return (uint32_t)(((1ull << 32) + d - 1) / d);
}

// Geometry of the streaming mat-vec (gemv_stream.cuh).
// variant = thr_code * 1000 + seg_code * 100 + tile_code * 10 + cap_code, -1 = default.
// `behind`: bytes of shared memory kept free behind the ring, taken from it.
bool plan_stream(long long n_out, int nb, int variant, StreamParams &p, int &threads, int &smem_bytes, int behind = 0) {
    if (nb % 2 != 0) return false;                  // rows must start on a word boundary
    int seg = 8 * STREAM_STEPS, tile_kb = 16, cap_kb = 108;
    threads = 512;
    if (variant >= 0) {
        static const int thr[] = {512, 384, 256, 128};
        static const int segs[] = {40, 32, 24, 16, 8, 40, 40, 40};
        static const int tiles[] = {16, 8, 12, 24, 32, 48, 6, 4};
        static const int caps[] = {108, 200, 72, 150};
        threads = thr[(variant / 1000) & 3];
        seg = segs[(variant / 100) % 10 & 7];
        tile_kb = tiles[(variant / 10) % 10 & 7];
        cap_kb = caps[variant % 10 & 3];
    }
    auto round_up = [](long long v, long long m) { return (v + m - 1) / m * m; };
    long long ctas = (n_out + 3) / 4;
    if (ctas > SM_COUNT) ctas = SM_COUNT;
    long long rows = round_up((n_out + ctas - 1) / ctas, 4);
    p.n_out = (int)n_out;
    p.nb = nb;
    const size_t row_bytes = (size_t)nb * W_BLOCK_BYTES;
    // segments: equal multiples of 8 blocks (every block lane of a task gets the same count), at most
    // what a task holds in registers
    p.nseg = (nb + seg - 1) / seg;
    p.seg_blocks = (int)round_up((nb + p.nseg - 1) / p.nseg, 8);
    if (p.seg_blocks > 8 * STREAM_STEPS) p.seg_blocks = 8 * STREAM_STEPS;
    p.nseg = (nb + p.seg_blocks - 1) / p.seg_blocks;
    for (int attempt = 0;; ++attempt) {
        const size_t fixed = 2 * RING_MAX_TILES * 8 + (size_t)nb * (STREAM_ACT_WORDS * 4 + 32) +
                             (size_t)rows * p.nseg * 4 + (size_t)((rows / 4 + 3) & ~3) * 4 + 16 + (size_t)behind;
        if ((size_t)cap_kb * 1024 < fixed + 64) return false;
        const size_t room = (size_t)cap_kb * 1024 - fixed - 64;
        long long tr = ((long long)tile_kb * 1024 / (long long)row_bytes) & ~3ll;
        if (tr < 4) tr = 4;
        if (tr > rows) tr = rows;
        while (tr > 4 && 3 * ((size_t)tr * row_bytes + 16) > room) tr -= 4;
        if (2 * ((size_t)tr * row_bytes + 16) > room) return false;
        long long nslot = (long long)(room / ((size_t)tr * row_bytes + 16));
        if (nslot > RING_MAX_SLOTS) nslot = RING_MAX_SLOTS;
        const long long ntiles = (rows + tr - 1) / tr;
        if (ntiles > RING_MAX_TILES) {          // very tall matrix: more CTAs, each with fewer rows
            if (attempt > 64) return false;
            const long long k = attempt + 2;
            rows = round_up((n_out + SM_COUNT * k - 1) / (SM_COUNT * k), 4);
            continue;
        }
        p.rows_per_cta = (int)rows;
        p.tr = (int)tr;
        p.nslot = (int)nslot;
        p.tpt = (p.tr / 4) * p.nseg;
        p.magic_tpt = magic_u32((uint32_t)p.tpt);
        p.magic_nseg = magic_u32((uint32_t)p.nseg);
        p.magic_nslot = magic_u32((uint32_t)p.nslot);
        smem_bytes = (int)(fixed + (size_t)p.nslot * ((size_t)tr * row_bytes + 16) + 64);
        return true;
    }
}

// Geometry of the tensor-core mat-vec (gemv_mma.cuh): tiles of 16 rows x one row segment, a ring of slots as deep
// as `cap_kb` of shared memory allows.  Rows must start on a word (nb even); rows longer than one segment are cut at
// multiples of 8 blocks (16-byte aligned pieces), which needs nb % 8 == 0.
bool plan_mma(long long n_out, int nb, int cap_kb, MmaGeom &P, int &smem_bytes, int &grid) {
    if (nb <= 0 || nb % 2 != 0) return false;
    P = MmaGeom{};
    P.n_out = (int)n_out;
    P.nb = nb;
    P.ngroups = (int)((n_out + 15) / 16);
    int seg_max;
    if (nb % 8 == 0) {
        const int units = nb / 8;
        P.nseg = (nb + MMA_SEG_MAX - 1) / MMA_SEG_MAX;
        P.seg_q = units / P.nseg;
        P.seg_r = units % P.nseg;
        seg_max = 8 * (P.seg_q + (P.seg_r ? 1 : 0));
    } else {
        if (nb > MMA_SEG_MAX + 8) return false;
        P.nseg = 1;
        seg_max = nb;
    }
    P.pairs_max = seg_max / 2;
    const int row_bytes = nb * W_BLOCK_BYTES;
    if (nb % 8 == 0) {
        // rows of a tile 16 * (odd) bytes apart: the 8 rows a load instruction touches fall into 8 different bank groups
        int stride = seg_max * W_BLOCK_BYTES;
        if ((stride / 16) % 2 == 0) stride += 16;
        P.contiguous = (P.nseg == 1 && stride == row_bytes) ? 1 : 0;
        P.stride = stride;
    } else {
        P.contiguous = 1;
        P.stride = row_bytes;
    }
    P.slot_bytes = (16 * P.stride + 127) & ~127;
    auto fixed = [&](int n) { return mma_fixed_bytes(P, n); };
    int nslot = MMA_MAX_SLOTS;
    while (nslot >= 2 && fixed(nslot) + (size_t)nslot * P.slot_bytes > (size_t)cap_kb * 1024) --nslot;
    if (nslot < 2) return false;
    P.nslot = nslot;
    P.magic_pairs = magic_u32((uint32_t)P.pairs_max);
    P.magic_nseg = magic_u32((uint32_t)P.nseg);
    P.magic_nslot = magic_u32((uint32_t)P.nslot);
    smem_bytes = (int)(fixed(nslot) + (size_t)nslot * P.slot_bytes);
    grid = P.ngroups < SM_COUNT ? P.ngroups : SM_COUNT;
    return true;
}

// Geometry of the small-batch mat-mul (gemv_mma.cuh, gemm_mma_kernel): tiles of 16 rows x one segment of at most
// MMAB_SEG_UNITS * 8 blocks, brought by one tiled copy when rows are a multiple of 8 blocks (16-byte aligned segment
// starts, row pitch a multiple of 16), else whole rows by one bulk copy (rows of at most 48 blocks).
bool plan_mmab(long long n_out, int nb, int n_tok, int cap_kb, MmabGeom &P, int &smem_bytes, int &grid) {
    if (nb <= 0 || nb % 2 != 0 || n_tok < 1 || n_tok > 16) return false;
    P = MmabGeom{};
    P.ntg = n_tok > 8 ? 2 : 1;
    // The segments and the items fix the order in which a row's terms are added: they depend on the row's length and
    // the token count only, never on n_out, so that a row slice gives the bits of the whole matrix.
    const int seg_units = P.ntg == 2 ? 1 : (nb >= 64 ? MMAB_SEG_UNITS : 2);
    // Two row groups per tile (a chunk's activation and header loads serve two MMAs) pay when a CTA has enough groups
    // to keep its warps busy with tiles of twice the size, and when the ring stays deep (16-block segments): measured
    // 172 -> 160 us on 5120 x 248320; with 2 .. 3 groups per CTA (17408 x 5120) 23 -> 29 us.
    P.nrg = (P.ntg == 1 && seg_units == 2 && (n_out + 15) / 16 >= 6ll * SM_COUNT) ? 2 : 1;
    P.n_out = (int)n_out;
    P.nb = nb;
    P.ngroups = (int)((n_out + 15) / 16);
    int seg_max;
    if (nb % 8 == 0) {
        const int units = nb / 8;
        P.nseg = (units + seg_units - 1) / seg_units;
        P.seg_q = units / P.nseg;
        P.seg_r = units % P.nseg;
        seg_max = 8 * (P.seg_q + (P.seg_r ? 1 : 0));
        int s16 = seg_max * W_BLOCK_BYTES / 16;         // rows of a tile 16 * (odd) bytes apart
        if (s16 % 2 == 0) ++s16;
        P.stride = 16 * s16;
        P.tiled = 1;
    } else {
        if (nb > 48 || P.ntg > 1) return false;
        P.nseg = 1;
        seg_max = nb;
        P.stride = nb * W_BLOCK_BYTES;
        P.tiled = 0;
    }
    P.pairs_max = seg_max / 2;
    P.ppi = P.ntg == 2 ? 1 : 2;                         // an item is 16 MMAs
    P.items = (P.pairs_max + P.ppi - 1) / P.ppi;
    P.slot_bytes = (P.nrg * 16 * P.stride + 127) & ~127;
    P.act_bufs = P.nseg > 1 ? 3 : 1;
    P.act_tab_off = (seg_max * 4 * n_tok * 36 + 8 * P.ntg * 36 + 127) & ~127;       // + what lanes past n_tok read beyond the last block
    P.act_buf_bytes = P.act_tab_off + seg_max * 4 * 64 * P.ntg;
    int nslot = MMA_MAX_SLOTS;
    while (nslot >= 2 && mmab_fixed_bytes(P, nslot) + (size_t)nslot * P.slot_bytes > (size_t)cap_kb * 1024) --nslot;
    if (nslot < 2) return false;
    P.nslot = nslot;
    P.magic_nslot = magic_u32((uint32_t)nslot);
    P.magic_bt = magic_u32((uint32_t)(MMAB_GB / P.nrg * P.nseg));
    P.magic_items = magic_u32((uint32_t)P.items);
    // tile and step numbers stay small enough for the multiplicative divisions of the kernel
    const long long groups_per_cta = (P.ngroups + SM_COUNT - 1) / SM_COUNT;
    if (groups_per_cta * P.nseg * P.items >= (1 << 24) || (groups_per_cta / MMAB_GB + 1) * P.nseg >= 65536) return false;
    smem_bytes = (int)(mmab_fixed_bytes(P, nslot) + (size_t)nslot * P.slot_bytes);
    grid = P.ngroups < SM_COUNT ? P.ngroups : SM_COUNT;
    return true;
}

// Geometry of the ring mat-vec: one CTA per SM, tiles of about 16 rows by one row segment, a ring that
// keeps the CTA under half of an SM's shared memory.
// variant = thr_code * 100000 + rr_code * 10000 + seg_code * 1000 + rs_code * 100 + chain_code * 10 + cap_code,
// -1 = default.
bool plan_ring(long long n_out, int npairs, int variant, RingParams &p, int &threads, int &smem_bytes, int &rr) {
    rr = 2;
    int seg_pairs = 16, rs_target = 16, chain = 3, cap_kb = 108;
    threads = 1024;
    if (variant >= 0) {
        static const int rrs[] = {1, 2, 4, 2};
        static const int segs[] = {16, 12, 20, 24, 32, 8, 1 << 20, 16};
        static const int rst[] = {16, 8, 32, 12, 24, 4, 16, 16};
        static const int chains[] = {3, 5, 1, 7};    // odd: with the copy warp an even count of warps computes
        static const int caps[] = {108, 200, 72, 150};
        rr = rrs[(variant / 10000) & 3];
        seg_pairs = segs[(variant / 1000) % 10 & 7];
        rs_target = rst[(variant / 100) % 10 & 7];
        chain = chains[(variant / 10) % 10 & 3];
        cap_kb = caps[variant % 10 & 3];
        static const int thr[] = {1024, 512, 768, 256};
        threads = thr[(variant / 100000) & 3];
    }
    if (rr == 4 && threads > 512) threads = 512;        // register budget of the four-row variant
    auto round_up = [](long long v, long long m) { return (v + m - 1) / m * m; };
    const int granule = npairs % 4 == 0 ? 1 : (npairs % 2 == 0 ? 2 : 4);      // rows per 16-byte aligned run
    const int unit = granule > rr ? granule : rr;
    long long ctas = (n_out + unit - 1) / unit;
    if (ctas > SM_COUNT) ctas = SM_COUNT;
    long long rows = round_up((n_out + ctas - 1) / ctas, unit);
    // a CTA has RING_MAX_TILES single-use barrier pairs: very tall matrices take more CTAs per SM
    const long long nseg_est = (npairs % 4 == 0 && npairs >= 2 * seg_pairs) ? npairs / seg_pairs : 1;
    const long long max_rows = (RING_MAX_TILES / nseg_est) * unit;      // tiles hold at least `unit` rows
    if (rows > max_rows) {
        const long long k = (n_out + max_rows * SM_COUNT - 1) / (max_rows * SM_COUNT);
        rows = round_up((n_out + SM_COUNT * k - 1) / (SM_COUNT * k), unit);
    }
    p.n_out = (int)n_out;
    p.npairs = npairs;
    p.rows_per_cta = (int)rows;
    if (npairs % 4 == 0 && npairs >= 2 * seg_pairs) {
        p.seg_base = seg_pairs;
        p.nseg = npairs / seg_pairs;
        p.sp = npairs - (p.nseg - 1) * seg_pairs;
        p.sw = 17 * p.sp;
        if ((p.sw / 4) % 2 == 0) p.sw += 4;            // odd count of 16-byte units: rows spread over 8 bank groups
    } else {
        p.nseg = 1;
        p.seg_base = p.sp = npairs;
        p.sw = 17 * npairs;
    }
    const size_t fixed = RING_BAR_BYTES + (size_t)npairs * ACT_REC_WORDS * 4;
    const size_t room = (size_t)cap_kb * 1024 > fixed + 64 ? (size_t)cap_kb * 1024 - fixed - 64 : 0;
    p.ts = 8 * p.sp + 4;                                   // an odd count of 16-byte units per row
    p.ntb = 3;
    long long rs = rs_target < rows ? round_up((rows + (rows + rs_target - 1) / rs_target - 1) /
                                               ((rows + rs_target - 1) / rs_target), unit)
                                    : rows;
    if (rs > 32) rs = 32 / unit * unit;
    auto need = [&](long long r, int slots) { return (size_t)r * ((size_t)p.sw * 4 * slots + (size_t)p.ts * 4 * p.ntb); };
    while (rs > unit && need(rs, 3) > room) rs -= unit;                 // three weight slots at least
    if (need(rs, 2) > room || rs < unit) return false;
    p.rs = (int)rs;
    long long nslot = (long long)((room - (size_t)rs * p.ts * 4 * p.ntb) / ((size_t)rs * p.sw * 4));
    if (nslot > RING_MAX_SLOTS) nslot = RING_MAX_SLOTS;
    p.nslot = (int)nslot;
    p.chain_warps = chain;
    if (((rows + p.rs - 1) / p.rs) * p.nseg > RING_MAX_TILES) return false;
    p.ppt = (p.rs / rr) * p.sp;
    p.magic_ppt = magic_u32((uint32_t)p.ppt);
    p.magic_sp = magic_u32((uint32_t)p.sp);
    p.magic_nseg = magic_u32((uint32_t)p.nseg);
    p.magic_nslot = magic_u32((uint32_t)p.nslot);
    p.magic_ntb = magic_u32((uint32_t)p.ntb);
    smem_bytes = (int)(fixed + need(p.rs, p.nslot) + 64);
    return true;
}

// Geometry of the staged mat-vec kernels.  `row_bytes` is the row stride, `fixed` the shared
// memory that does not depend on the row count, `granule` the row multiple that keeps a run of
// rows 16-byte aligned.  CTA counts are multiples of the SM count, so every SM gets the same
// share, and a CTA stays under half of an SM's shared memory so that a second CTA -- of this launch
// or, with programmatic launches, of the next kernel in the stream -- can stream beside it.
GemvPlan plan_rows(long long n_out, size_t row_bytes, size_t fixed, int granule, int variant) {
    // variant = rr_code * 1000 + cap_code * 100 + stage_code * 10 + thread_code, or -1 = tuned default
    int rr = 2, cap_kb = 111, stage_kb = 8, threads = 512;
    if (variant >= 0) {
        static const int rrs[] = {1, 2, 4, 2};
        static const int caps[] = {111, 220, 72, 56};
        static const int stages[] = {4, 8, 12, 16, 24, 32, 48, 64};
        static const int thr[] = {256, 512, 1024, 384};
        rr = rrs[(variant / 1000) & 3];
        cap_kb = caps[(variant / 100) % 10 & 3];
        stage_kb = stages[(variant / 10) % 10 & 7];
        threads = thr[variant % 10 & 3];
    }
    if (rr == 4 && threads > 512) threads = 512;       // register budget of the four-row variant
    const int unit = granule > rr ? granule : rr;      // both are powers of two
    auto round_up = [](long long v, long long m) { return (v + m - 1) / m * m; };
    const size_t room = (size_t)cap_kb * 1024 - GEMV_BAR_BYTES - fixed - 64;
    long long rows = unit;
    for (int k = 1;; ++k) {
        const long long ctas = (long long)SM_COUNT * k;
        rows = round_up((n_out + ctas - 1) / ctas, unit);
        if ((size_t)rows * row_bytes <= room || rows == unit) break;
    }
    GemvPlan p;
    p.rr = rr;
    p.threads = threads;
    p.rows_per_cta = (int)rows;
    p.ctas = (int)((n_out + rows - 1) / rows);
    long long rps = round_up(((long long)stage_kb * 1024 + row_bytes - 1) / row_bytes, unit);
    const long long min_rps = round_up((rows + GEMV_MAX_STAGES - 1) / GEMV_MAX_STAGES, unit);
    if (rps < min_rps) rps = min_rps;
    p.rows_per_stage = (int)rps;
    // chain warps come in twos (compute warps must stay paired), at most a quarter of the CTA
    int chain = 2 * (int)((rows + 63) / 64);
    const int max_chain = threads / 32 / 4 >= 2 ? (threads / 32 / 4) & ~1 : 2;
    p.chain_warps = chain < max_chain ? chain : max_chain;
    p.smem_bytes = (int)(GEMV_BAR_BYTES + fixed + (size_t)rows * row_bytes + 64);
    return p;
}

// Any float pointers are taken, as by the reference; 16-byte aligned ones get 16-byte accesses.
int launch_fwht(bool vec, const float *x, const float *signs, float *x_rot, void *xq, int64_t n_in, int64_t n_tok, bonsai_stream stream) {
    const long long blocks = (n_in / FWHT_N) * n_tok;
    if (blocks > INT32_MAX) return 1;
    // A CTA per block for few blocks (a short chain, eight warps on it), a warp per block for many (a third of the instructions).  The line, in blocks per SM,
    // with the times on both sides: 2 with the quantiser (200 blocks: 2.29 us and 2.34, 340 2.78 and 2.68, 500 3.22 and 2.56; in front of their mat-mul 240 22.35
    // and 22.65, 340 34.5 and 33.5), 1 for the rotation alone (120: 1.89 and 2.00, 200: 2.18 and 1.84).  The same lines serve vectors that are stored as well and 4-byte accesses (replayed by a
    // graph: with quantiser and stored 250 blocks 2.18 and 2.49, 300 2.59 and 2.63, 400 2.63 and 2.73, 600 4.44 and 3.21, 1800 6.93 and 5.09; by 4 bytes 250 2.39 and 2.63, 300 2.83 and 2.80, 400 2.90
    // and 2.83, 600 4.57 and 3.41, 1800 7.85 and 5.80; both 400 3.04 and 2.93, 1800 8.47 and 6.18, 10000 40.9 and 26.9; rotation by 4 bytes 160 2.29 and 2.32, 300 2.53 and 2.46, 1800 7.31 and 4.98).
    const bool warps = blocks > (long long)SM_COUNT * (xq ? 2 : 1);
    return (int)launch(warps ? (vec ? fwht_quant_warp_kernel<true> : fwht_quant_warp_kernel<false>) : (vec ? fwht_quant_kernel<true> : fwht_quant_kernel<false>),
                       dim3((unsigned)blocks), dim3(warps ? 32 : FWHT_THREADS), 0, as_stream(stream), true, x, signs, x_rot, static_cast<uint32_t *>(xq), (int)n_in, (int)n_tok);
}

int launch_quant(bool vec, const float *X, void *Xq, int64_t n_in, int64_t n_tok, long long blocks, bonsai_stream stream) {
    auto run = [&](auto kernel) {
        return (int)launch(kernel, dim3((unsigned)blocks), dim3(256), 0, as_stream(stream), true, X, static_cast<uint32_t *>(Xq), (int)n_in, (int)n_tok);
    };
    if (blocks <= SM_COUNT) return vec ? run(quant_q8_1_kernel<true, true>) : run(quant_q8_1_kernel<false, true>);
    return vec ? run(quant_q8_1_kernel<true, false>) : run(quant_q8_1_kernel<false, false>);
}

}  // namespace

extern "C" {

int bonsai_p40_quant_activations(const float *x, void *out, int64_t n, bonsai_stream stream) {
    if (n <= 0 || n % 32 != 0) return 1;
    if (!aligned4(x) || !aligned4(out) || n > INT32_MAX) return 1;
    const long long threads = n / 4;
    const int blocks = (int)((threads + 255) / 256);
    // any float pointer is taken, as by the reference; 16-byte aligned ones get 16-byte loads
    return launch_quant(aligned16(x), x, out, n, 1, blocks, stream);
}

int bonsai_p40_fwht(float *x, const float *signs, int64_t n, bonsai_stream stream) {
    if (n <= 0 || n % FWHT_N != 0) return 1;
    if (!aligned4(x) || (signs && !aligned4(signs)) || n > INT32_MAX) return 1;
    return launch_fwht(aligned16(x) && (!signs || aligned16(signs)), x, signs, x, nullptr, n, 1, stream);
}

int bonsai_b200_fwht_quant(const float *x, const float *signs, void *xq, float *x_rot, int64_t n,
                           bonsai_stream stream) {
    if (n <= 0 || n % FWHT_N != 0 || n > INT32_MAX) return 1;
    if (!aligned4(x) || (signs && !aligned4(signs)) || (x_rot && !aligned4(x_rot)) || !aligned4(xq)) return 1;
    return launch_fwht(aligned16(x) && (!signs || aligned16(signs)) && (!x_rot || aligned16(x_rot)), x, signs, x_rot, xq, n, 1, stream);
}

int bonsai_b200_quant_batch(const float *X, const float *signs, void *Xq, int64_t n_in, int64_t n_tok, int rotate,
                            bonsai_stream stream) {
    if (n_in <= 0 || n_tok <= 0 || n_in % 32 != 0) return 1;
    if (rotate && n_in % FWHT_N != 0) return 1;
    if (!aligned4(X) || (signs && !aligned4(signs)) || !aligned4(Xq)) return 1;
    if (n_in > INT32_MAX || n_tok > INT32_MAX) return 1;
    const bool vec = aligned16(X) && (!signs || aligned16(signs));
    if (rotate) {
        return launch_fwht(vec, X, signs, nullptr, Xq, n_in, n_tok, stream);
    }
    const long long threads = n_in / 4 * n_tok;
    long long blocks = (threads + 255) / 256;
    if (blocks > 8 * SM_COUNT * 4) blocks = 8 * SM_COUNT * 4;
    return launch_quant(vec, X, Xq, n_in, n_tok, blocks, stream);
}

// behind_quantiser: the launch before this one on the stream is this library's quantiser, so nothing that is still running
// writes the weights and the first tiles are copied before the wait for it.
static int gemv_launch(const void *W, const void *xq, float *y, int64_t n_out, int64_t n_in, bonsai_stream stream, bool behind_quantiser) {
    if (n_in <= 0 || n_in % 128 != 0) return 1;
    if (n_out <= 0) return 0;
    if (n_out > INT32_MAX || n_in / 128 > INT32_MAX / 64) return 1;
    const int nblocks = (int)(n_in / 128);
    const bool pdl = g_opt_pdl.load() != 0;
    const int variant = g_opt_gemv_variant.load();
    const bool base_ok = (nblocks % 2 == 0) && aligned16(W) && !(reinterpret_cast<uintptr_t>(xq) & 3u);
    int threads = 0, smem_bytes = 0, rr = 2;
    if (g_opt_gemv_order.load() == 2) {
        MmaGeom mp;
        int grid = 0;
        if (base_ok && plan_mma(n_out, nblocks, 200, mp, smem_bytes, grid)) {
            static SmemOptIn opt;
            cudaError_t err = opt.ensure(gemv_mma_kernel<false>);
            if (err != cudaSuccess) return (int)err;
            return (int)launch(gemv_mma_kernel<false>, dim3((unsigned)grid), dim3(MMA_THREADS), (size_t)smem_bytes,
                               as_stream(stream), pdl, static_cast<const uint8_t *>(W), static_cast<const uint32_t *>(xq), y,
                               mp, static_cast<int32_t *>(nullptr));
        }
    }
    if (g_opt_gemv_order.load() != 1) {
        StreamParams sp;
        if (base_ok && plan_stream(n_out, nblocks, variant, sp, threads, smem_bytes)) {
            static SmemOptIn opt;
            cudaError_t err = opt.ensure(gemv_stream_kernel<false>);
            if (err != cudaSuccess) return (int)err;
            sp.early = pdl || behind_quantiser;
            return (int)launch(gemv_stream_kernel<false>, dim3((unsigned)((n_out + sp.rows_per_cta - 1) / sp.rows_per_cta)),
                               dim3(threads), (size_t)smem_bytes, as_stream(stream), true,
                               static_cast<const uint8_t *>(W), static_cast<const uint32_t *>(xq), y, sp,
                               static_cast<const float *>(nullptr), static_cast<const float *>(nullptr),
                               static_cast<uint32_t *>(nullptr));
        }
    }
    RingParams rp;
    const bool ring = base_ok && g_opt_gemv_order.load() == 1 &&
                      plan_ring(n_out, nblocks / 2, variant, rp, threads, smem_bytes, rr);
    if (!ring) {
        // odd block count, unaligned weights or a row too long for the rings: plain loads, host order
        return (int)launch(gemv_pq2_generic_kernel, dim3((unsigned)((n_out + 7) / 8)), dim3(256), 0, as_stream(stream),
                           pdl, static_cast<const uint8_t *>(W), static_cast<const uint8_t *>(xq), y, (int)n_out,
                           nblocks);
    }
    const dim3 grid((unsigned)((n_out + rp.rows_per_cta - 1) / rp.rows_per_cta));
    static SmemOptIn opt1, opt2, opt4;
    auto go = [&](auto kernel, SmemOptIn &opt) -> cudaError_t {
        cudaError_t err = opt.ensure(kernel);
        if (err != cudaSuccess) return err;
        return launch(kernel, grid, dim3(threads), (size_t)smem_bytes, as_stream(stream), pdl,
                      static_cast<const uint8_t *>(W), static_cast<const uint32_t *>(xq), y, rp);
    };
    cudaError_t e;
    if (rr == 1) e = go(gemv_ring_kernel<1>, opt1);
    else if (rr == 2) e = go(gemv_ring_kernel<2>, opt2);
    else e = go(gemv_ring_kernel<4>, opt4);
    return (int)e;
}

int bonsai_p40_gemv(const void *W, const void *xq, float *y, int64_t n_out, int64_t n_in, bonsai_stream stream) {
    return gemv_launch(W, xq, y, n_out, n_in, stream, false);
}

// One projection in one launch, rotation and quantiser in the prologue of the streaming mat-vec.  -1: two launches serve.
static int linear_one_launch(const void *W, const float *x, const float *signs, float *y, void *xq, int64_t n_out, int64_t n_in, bonsai_stream stream) {
    const int fuse = g_opt_fuse_linear.load();
    if (g_opt_gemv_order.load() != 0 || fuse == 0 || !aligned16(W) || !aligned16(x) || (signs && !aligned16(signs)) || n_out > INT32_MAX || n_in > INT32_MAX) return -1;
    // (of two launches the second may overwrite what the first has read: here CTAs still read it)
    auto apart = [&](const float *p) {
        const auto lo = reinterpret_cast<uintptr_t>(p), hi = lo + 4 * (uintptr_t)n_in, y0 = reinterpret_cast<uintptr_t>(y), q0 = reinterpret_cast<uintptr_t>(xq);
        return !p || ((hi <= y0 || y0 + 4 * (uintptr_t)n_out <= lo) && (hi <= q0 || q0 + (uintptr_t)n_in / 32 * A_BLOCK_BYTES <= lo));
    };
    if (!apart(x) || !apart(signs)) return -1;
    const int nb = (int)(n_in / 128), nfb = nb / 8;
    StreamParams sp;
    int threads = 0, smem_bytes = 0;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.stream = as_stream(stream);
    const uint8_t *w8 = static_cast<const uint8_t *>(W);
    uint32_t *blocks = static_cast<uint32_t *>(xq);
    // The kernel for few rows: as few row quads per CTA as let every CTA find an SM of its own, at most two pieces per warp.  Clusters of nfb CTAs
    // of which two fit an SM are packed two to an SM from FEW_ALONE[nfb] of them on (us for that many and for one more: 3072 wide 3.35 and 4.00, 4096
    // 3.31 and 3.68, 5120 3.52 and 3.85, 6144 4.04 and 4.60, 7168 4.18 and 5.24).  us, two launches / one (calls; with a graph's replay): 1024 -> 64 3.96 / 2.70 (3.26 /
    // 2.45), -> 4096 4.36 / 3.03; 3072 -> 1500 4.80 / 3.45; 5120 -> 64 4.54 / 3.24 (3.78 / 3.04), -> 1024 4.92 / 3.91 (3.88 / 3.68), -> 1850 5.38 / 4.10;
    // 6144 -> 1000 5.15 / 4.22; 8192 -> 600 5.48 / 4.44.  With more pieces per warp, two blocks per CTA or CTAs two to an SM a graph's replay of two launches
    // is ahead: 5120 -> 3000 5.70 / 5.61 (4.84 / 5.28), 9216 -> 600 5.54 / 5.00 (4.40 / 4.80), 4096 -> 1500 in 32 clusters 5.07 / 4.41 (3.90 / 4.18).
    if (nfb <= FEW_MAX_CLUSTER && plan_stream(n_out, nb, g_opt_gemv_variant.load(), sp, threads, smem_bytes)) {
        static const int FEW_ALONE[FEW_MAX_CLUSTER + 1] = {0, SM_COUNT, 74, 44, 24, 24, 15, 15, 15};
        const int room = nfb == 1 ? SM_COUNT : g_few_clusters[nfb].ask(gemv_few_kernel<FEW_HELD>, g_few_opt[FEW_HELD - 1], (unsigned)nfb, 32 * FEW_WARPS);
        const long long most = std::min(room, FEW_ALONE[nfb]), quads_in_all = (n_out + 3) / 4;
        const long long need = most > 0 ? (quads_in_all + most * nfb - 1) / (most * nfb) : FEW_HELD * FEW_WARPS + 1;
        if (need * nfb <= (nfb == 1 ? 1 : FEW_HELD) * FEW_WARPS) {
            const int quads = (int)need;
            const unsigned clusters = (unsigned)((quads_in_all + (long long)quads * nfb - 1) / ((long long)quads * nfb));
            attr[0].val.clusterDim.x = (unsigned)nfb;
            cfg.gridDim = dim3(clusters * (unsigned)nfb);
            cfg.blockDim = dim3(32 * FEW_WARPS);
            cfg.dynamicSmemBytes = (size_t)few_smem_bytes(nb, quads, sp.nseg);
            cfg.attrs = nfb == 1 ? attr + 1 : attr;
            cfg.numAttrs = (nfb > 1) + (g_opt_overlap.load() != 0);
            auto go = [&](auto kernel, SmemOptIn &o) -> cudaError_t {
                const cudaError_t err = o.ensure(kernel);
                if (err != cudaSuccess) return err;
                const int rows = (int)n_out, seg_steps = sp.seg_blocks / 8;
                return nfb > 1 ? launch_clusters(cfg, kernel, w8, x, signs, y, blocks, rows, nb, seg_steps, quads) : cudaLaunchKernelEx(&cfg, kernel, w8, x, signs, y, blocks, rows, nb, seg_steps, quads);
            };
            const cudaError_t err = quads * nfb <= FEW_WARPS ? go(gemv_few_kernel<1>, g_few_opt[0]) : go(gemv_few_kernel<2>, g_few_opt[1]);
            if (nfb == 1 || !g_few_clusters[nfb].refused(err)) return (int)err;
        }
    }
    // One block of 1024, whatever the rows: every CTA rotates it for itself (us, two launches / one: -> 10240 5.27 / 4.40, -> 40000 8.51 / 7.54; 2048 wide a graph's
    // replay of two launches is ahead: -> 17408 6.97 / 6.50 (5.84 / 6.05), 5120 wide calls are too: -> 17408 10.91 / 12.17).
    if (fuse < 0 && nfb > 1) return -1;
    if (!plan_stream(n_out, nb, g_opt_gemv_variant.load(), sp, threads, smem_bytes, std::min(nfb, LIN_BLOCKS) * FWHT_N * 4) || threads != 512) return -1;
    sp.early = g_opt_pdl.load() != 0;
    static SmemOptIn opt;
    const cudaError_t err = opt.ensure(gemv_stream_kernel<true>);
    if (err != cudaSuccess) return (int)err;
    return (int)launch(gemv_stream_kernel<true>, dim3((unsigned)((n_out + sp.rows_per_cta - 1) / sp.rows_per_cta)), dim3(threads), (size_t)smem_bytes, as_stream(stream),
                       true, w8, static_cast<const uint32_t *>(nullptr), y, sp, x, signs, blocks);
}

static int linear_launch(const void *W, const float *x, const float *signs, float *y, void *xq, int64_t n_out, int64_t n_in, bonsai_stream stream) {
    const int one = linear_one_launch(W, x, signs, y, xq, n_out, n_in, stream);
    if (one >= 0) return one;
    const int rc = bonsai_b200_fwht_quant(x, signs, xq, nullptr, n_in, stream);
    if (rc != 0) return rc;
    return gemv_launch(W, xq, y, n_out, n_in, stream, true);
}

int bonsai_b200_linear(const void *W, const float *x, const float *signs, float *y, void *xq_scratch, int64_t n_out,
                       int64_t n_in, bonsai_stream stream) {
    if (n_out <= 0 || n_in <= 0 || n_in % FWHT_N != 0 || !xq_scratch) return 1;
    if (n_out > INT32_MAX || !aligned4(x) || (signs && !aligned4(signs)) || !aligned4(xq_scratch)) return 1;
    return linear_launch(W, x, signs, y, xq_scratch, n_out, n_in, stream);
}

// ---- projection without any allocation: the Q8_1 scratch is part of the library image -----------
// In host code the array's name is only a handle: the device address comes from
// cudaGetSymbolAddress, once per device, with that device current.
static __device__ __align__(256) unsigned char g_linear_static_xq[BONSAI_B200_LINEAR_STATIC_MAX_N_IN / 32 * A_BLOCK_BYTES];

int bonsai_b200_linear_static(const void *W, const float *x, const float *signs, float *y, int64_t n_out, int64_t n_in,
                              bonsai_stream stream) {
    if (n_in > BONSAI_B200_LINEAR_STATIC_MAX_N_IN) return BONSAI_B200_ETOOLARGE;
    if (n_out <= 0 || n_in <= 0 || n_in % FWHT_N != 0) return 1;
    constexpr int MAX_DEVICES = 64;
    static std::atomic<void *> scratch_of_device[MAX_DEVICES];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= MAX_DEVICES) return 1;
    void *scratch = scratch_of_device[dev].load(std::memory_order_acquire);
    if (!scratch) {     // first call on this device: resolve the device address of the array
        e = cudaGetSymbolAddress(&scratch, g_linear_static_xq);
        if (e != cudaSuccess) return (int)e;
        if (!scratch) return (int)cudaErrorInvalidSymbol;
        scratch_of_device[dev].store(scratch, std::memory_order_release);
    }
    return linear_launch(W, x, signs, y, scratch, n_out, n_in, stream);
}


// ---- a list of projections in one persistent launch ------------------------------------------------
struct bonsai_b200_chain {
    ChainOp *d_ops = nullptr;
    unsigned int *d_counter = nullptr;      // [0] arrivals of ops that others wait for
    uint8_t *d_image = nullptr;             // activation tables of a spread op, shared through L2 (one rank: behind the counters)
    bool tp = false;                        // several ranks: counters live in the caller's peer-mapped buffer, never reset
    ChainPeers peers{};
    int n_ops = 0, threads = 0, grid = 0, device = 0;
    size_t smem = 0, counter_bytes = 0;
    ChainGeom G{};
};

static int chain_create_impl(const bonsai_b200_op *ops, int64_t n_ops, int tp_rank, int tp_world,
                             const void *const *peer_base, int64_t buffer_bytes, int64_t counter_offset,
                             int64_t wait_limit_us, bonsai_b200_chain **out) {
    if (!ops || !out || n_ops <= 0 || n_ops > (1 << 20)) return 1;
    *out = nullptr;
    const bool tp = tp_world > 1;
    if (tp) {
        if (tp_world > CHAIN_MAX_RANKS || tp_rank < 0 || tp_rank >= tp_world || !peer_base || counter_offset < 0 ||
            (counter_offset & 63) || wait_limit_us < 0)
            return 1;
        // the counter block lies inside the buffer, behind every output; every mapping is 16-byte aligned
        if (buffer_bytes < counter_offset + BONSAI_B200_TP_COUNTER_BYTES) return 1;
        for (int q = 0; q < tp_world; ++q)
            if (!peer_base[q] || !aligned16(peer_base[q])) return 1;
        // every output must lie inside [buffer, counters): the kernel stores it at the same offset of every
        // rank's mapping, so an output outside the buffer would be a store into memory that is not ours
        const char *lo = static_cast<const char *>(peer_base[tp_rank]);
        for (int64_t i = 0; i < n_ops; ++i) {
            const char *y = reinterpret_cast<const char *>(ops[i].y);
            if (!y || ops[i].n_out <= 0 || y < lo || y + ops[i].n_out * 4 > lo + counter_offset) return 1;
        }
    }
    int dev = 0, sms = 0, smem_limit = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return (int)e;
    if ((e = cudaDeviceGetAttribute(&smem_limit, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) != cudaSuccess) return (int)e;
    if (sms <= 0) return 1;
    auto round_up = [](long long v, long long m) { return (v + m - 1) / m * m; };
    const long long tile_target = (long long)g_opt_chain_tile_kb.load() * 1024;
    const int threads_opt = g_opt_chain_threads.load();
    const int steps_max = threads_opt == 768 ? 3 : threads_opt == 640 ? 4 : STREAM_STEPS;
    const int seg_max = g_opt_chain_seg.load() < 8 * steps_max ? g_opt_chain_seg.load() : 8 * steps_max;

    std::vector<ChainOp> rec((size_t)n_ops);
    ChainGeom G{};
    long long slot_payload = 0;
    // Table buffers: a third one lets the sequencer prepare two inputs ahead, which pays when most ops bring
    // their own Q8_1 vector; lists whose ops mostly share inputs keep the shared memory for the ring instead.
    int q8_ops = 0, q8_fills = 0;
    for (int64_t i = 0; i < n_ops; ++i) {
        if (ops[i].flags & BONSAI_B200_OP_ROTATE) continue;
        ++q8_ops;
        const bool shared = (ops[i].flags & BONSAI_B200_OP_SAME_INPUT) ||
                            (i > 0 && ops[i - 1].x == ops[i].x && ops[i - 1].n_in == ops[i].n_in &&
                             !(ops[i - 1].flags & BONSAI_B200_OP_ROTATE));
        if (!shared) ++q8_fills;
    }
    // What the list writes, in order of address, each with the furthest end so far: norm weights or signs in there are read late.
    std::vector<std::pair<uintptr_t, uintptr_t>> written;
    for (int64_t i = 0; i < n_ops; ++i) {
        const uintptr_t y = reinterpret_cast<uintptr_t>(ops[i].y);
        if (ops[i].n_out > 0) written.emplace_back(y, y + 4 * (uintptr_t)ops[i].n_out);
    }
    if (tp) {                                                   // the other ranks write their rows here too
        const uintptr_t b = reinterpret_cast<uintptr_t>(peer_base[tp_rank]);
        written.emplace_back(b, b + (uintptr_t)counter_offset);
    }
    std::sort(written.begin(), written.end());
    for (size_t i = 1; i < written.size(); ++i) written[i].second = std::max(written[i].second, written[i - 1].second);
    auto list_writes = [&](const float *p, int64_t n) {
        const uintptr_t lo = reinterpret_cast<uintptr_t>(p), hi = lo + 4 * (uintptr_t)n;
        const auto behind = std::lower_bound(written.begin(), written.end(), std::make_pair(hi, (uintptr_t)0));   // the first that starts behind them
        return behind != written.begin() && std::prev(behind)->second > lo;
    };
    const int ntables = q8_ops == 0 ? 1 : (2 * q8_fills > q8_ops ? CHAIN_TABLES : 2);
    int shift = 0, buf = ntables - 1, last_user[CHAIN_TABLES], ready_uses[CHAIN_TABLES];
    for (int b = 0; b < CHAIN_TABLES; ++b) last_user[b] = -1, ready_uses[b] = 0;
    bool any_rotate = false, any_q8 = false, any_spread = false, any_rescale = false;
    unsigned int spread_total = 0;
    const int spread_nb = g_opt_chain_spread_nb.load();
    unsigned int signals = 0;
    for (int64_t i = 0; i < n_ops; ++i) {
        const bonsai_b200_op &o = ops[i];
        ChainOp &r = rec[(size_t)i];
        std::memset(&r, 0, sizeof(r));
        const bool rotate = o.flags & BONSAI_B200_OP_ROTATE, depends = o.flags & BONSAI_B200_OP_DEPENDS;
        bool same = o.flags & BONSAI_B200_OP_SAME_INPUT;
        const uint32_t producer = o.flags & (BONSAI_B200_OP_RMSNORM | BONSAI_B200_OP_SWIGLU | BONSAI_B200_OP_RESCALE);
        // two ops read the same prepared input: same vector, width, signs, kind and producer (with its arguments)
        auto same_input = [](const bonsai_b200_op &a, const bonsai_b200_op &b) {
            const uint32_t kind = BONSAI_B200_OP_ROTATE | BONSAI_B200_OP_RMSNORM | BONSAI_B200_OP_SWIGLU | BONSAI_B200_OP_RESCALE;
            return a.x == b.x && a.n_in == b.n_in && a.signs == b.signs && !((a.flags ^ b.flags) & kind) && a.aux == b.aux &&
                   a.eps == b.eps && a.src_len == b.src_len;
        };
        // the same vector as the op before, and no wait asked for: its tables are reused without being told
        // (nothing may write x during the launch unless a later reader says OP_DEPENDS)
        if (!same && i > 0 && !depends && same_input(ops[i - 1], o)) same = true;
        if ((o.flags & ~63u) || o.reserved) return 1;
        if (!o.W || !o.x || !o.y || o.n_out <= 0 || o.n_out > INT32_MAX || o.n_in <= 0) return 1;
        if (o.n_in % 256 != 0 || (rotate && o.n_in % FWHT_N != 0) || o.n_in / 128 > 1024) return 1;
        if (!aligned16(o.W) || !aligned16(o.x) || (o.signs && !aligned16(o.signs)) || (reinterpret_cast<uintptr_t>(o.y) & 3u))
            return 1;
        if (depends && !rotate) return 1;               // outputs are fp32: a dependent op must quantise
        if (o.signs && !rotate) return 1;
        // producers work on the fp32 vector, one at a time
        if (producer && (!rotate || (producer & (producer - 1)))) return 1;
        if ((producer & (BONSAI_B200_OP_RMSNORM | BONSAI_B200_OP_SWIGLU)) && (!o.aux || !aligned16(o.aux))) return 1;
        if (!(producer & (BONSAI_B200_OP_RMSNORM | BONSAI_B200_OP_SWIGLU)) && o.aux) return 1;
        if ((producer & BONSAI_B200_OP_RMSNORM) && o.n_in / FWHT_N > 7) return 1;      // the whole vector must fit one pass
        if (!(producer & BONSAI_B200_OP_RMSNORM) && o.eps != 0.0f) return 1;
        int src_op = -1;
        if (producer & BONSAI_B200_OP_RESCALE) {
            // x is the output of an earlier op of the list (all of it), whose largest magnitude the kernel records
            if (tp || o.src_len == 0 || o.src_len % 4 != 0 || o.src_len > INT32_MAX) return 1;
            for (int64_t pidx = i - 1; pidx >= 0 && src_op < 0; --pidx)
                if (ops[pidx].y == o.x && ops[pidx].n_out == (int64_t)o.src_len) src_op = (int)pidx;
            if (src_op < 0) return 1;
        } else if (o.src_len != 0) {
            return 1;
        }
        if (same) {
            if (i == 0 || depends) return 1;
            if (!same_input(ops[i - 1], o)) return 1;
        }
        r.W = static_cast<const uint8_t *>(o.W);
        r.x = o.x;
        r.signs = o.signs;
        r.y = o.y;
        r.nb = (int)(o.n_in / 128);
        r.n_out = (int)o.n_out;
        long long ctas = (o.n_out + 3) / 4;
        if (ctas > sms) ctas = sms;
        r.rows_per_cta = (int)round_up((o.n_out + ctas - 1) / ctas, 4);
        const long long used = (o.n_out + r.rows_per_cta - 1) / r.rows_per_cta;
        const long long row_bytes = (long long)r.nb * W_BLOCK_BYTES;
        long long tr = (tile_target / row_bytes) & ~3ll;
        if (tr < 4) tr = 4;
        if (tr > r.rows_per_cta) tr = r.rows_per_cta;
        r.tr = (int)tr;
        r.nseg = (r.nb + seg_max - 1) / seg_max;
        r.seg_blocks = (int)round_up((r.nb + r.nseg - 1) / r.nseg, 8);
        if (r.seg_blocks > seg_max) r.seg_blocks = seg_max;
        r.nseg = (r.nb + r.seg_blocks - 1) / r.seg_blocks;
        r.tpt = (r.tr / 4) * r.nseg;
        r.magic_tpt = magic_u32((uint32_t)r.tpt);
        r.magic_nseg = magic_u32((uint32_t)r.nseg);
        r.cta_shift = shift;
        shift = (int)((shift + used) % sms);            // the next op starts on the CTA after this one's last
        r.flags = (rotate ? CHAIN_ROTATE : 0) | (depends ? CHAIN_DEPENDS : 0) | (same ? CHAIN_SAME_INPUT : 0) |
                  ((producer & BONSAI_B200_OP_RMSNORM) ? CHAIN_RMSNORM : 0) | ((producer & BONSAI_B200_OP_SWIGLU) ? CHAIN_SWIGLU : 0) |
                  ((producer & BONSAI_B200_OP_RESCALE) ? CHAIN_RESCALE : 0);
        if (((producer & BONSAI_B200_OP_RMSNORM) && list_writes(o.aux, o.n_in)) || (o.signs && list_writes(o.signs, o.n_in))) r.flags |= CHAIN_LATE;
        r.aux = o.aux;
        r.eps = o.eps;
        r.src_len = (int)o.src_len;
        r.src_op = src_op;
        if (src_op >= 0) {
            rec[(size_t)src_op].flags |= CHAIN_MAXSRC;
            any_rescale = true;
        }
        if (depends) rec[(size_t)i - 1].flags |= CHAIN_SIGNAL;     // i > 0: op 0 may not depend
        if (depends && i == 0) return 1;
        if (!same) buf = (buf + 1) % ntables;
        r.buf = buf;
        r.prev_user = same ? -1 : last_user[buf];
        last_user[buf] = (int)i;
        if (!same && !rotate) r.ready_parity = ready_uses[buf]++ & 1;
        if (rotate) any_rotate = true; else any_q8 = true;
        if (rotate && depends && !same && spread_nb > 0 && r.nb >= spread_nb && r.nb / 8 <= sms) {
            r.flags |= CHAIN_SPREAD;
            spread_total += (unsigned)(r.nb / 8);
            r.spread_blocks = spread_total;
            any_spread = true;
        }
        if (r.nb > G.nb_max) G.nb_max = r.nb;
        if (r.nseg > 1) {        // only rows in several segments are joined through shared memory
            if (r.rows_per_cta * r.nseg > G.partial_floats) G.partial_floats = r.rows_per_cta * r.nseg;
            if (r.rows_per_cta / 4 > G.quad_ints) G.quad_ints = r.rows_per_cta / 4;
        }
        if (tr * row_bytes > slot_payload) slot_payload = tr * row_bytes;
    }
    if (tp) rec[(size_t)n_ops - 1].flags |= CHAIN_SIGNAL;       // the closing arrival of a run
    // arrivals a dependent op must see: one per CTA for every signalling op before it
    for (int64_t i = 0; i < n_ops; ++i) {
        rec[(size_t)i].arrivals_needed = signals;
        if (rec[(size_t)i].flags & CHAIN_SIGNAL) ++signals;
    }
    G.stage_blocks = any_q8 ? G.nb_max : 0;
    G.ntables = ntables;
    G.rot_blocks = any_rotate ? (G.nb_max / 8 < 7 ? G.nb_max / 8 : 7) : 0;
    if (tp)
        for (const auto &r : rec)
            if (r.rows_per_cta > G.rows_stage) G.rows_stage = r.rows_per_cta;
    G.partial_floats = (int)round_up(G.partial_floats, 4);
    G.quad_ints = (int)round_up(G.quad_ints, 4);
    G.slot_bytes = (int)round_up(slot_payload + 16, 128);
    const size_t fixed = chain_fixed_bytes(G);
    if (fixed + 3 * (size_t)G.slot_bytes > (size_t)smem_limit) return 1;
    long long nslot = ((long long)smem_limit - (long long)fixed) / G.slot_bytes;
    if (nslot > CHAIN_MAX_SLOTS) nslot = CHAIN_MAX_SLOTS;
    G.nslot = (int)nslot;
    G.magic_nslot = magic_u32((uint32_t)G.nslot);

    bonsai_b200_chain *c = new (std::nothrow) bonsai_b200_chain;
    if (!c) return (int)cudaErrorMemoryAllocation;
    c->n_ops = (int)n_ops;
    c->threads = threads_opt;
    c->tp = tp;
    if (tp) {
        if (threads_opt != 512) { delete c; return 1; }             // the several-rank kernel is built for 512 threads
        c->peers.rank = tp_rank;
        c->peers.world = tp_world;
        c->peers.arrivals_per_run = signals;
        c->peers.spread_per_run = spread_total;
        c->peers.wait_limit_ns = (unsigned long long)(wait_limit_us > 0 ? wait_limit_us : 1000000) * 1000ull;
        for (int q = 0; q < tp_world; ++q) {
            c->peers.y_delta[q] = (long long)(static_cast<const char *>(peer_base[q]) - static_cast<const char *>(peer_base[tp_rank]));
            c->peers.counter[q] = reinterpret_cast<unsigned int *>(const_cast<char *>(static_cast<const char *>(peer_base[q])) + counter_offset);
        }
    }
    c->grid = sms;
    c->device = dev;
    c->G = G;
    c->smem = fixed + (size_t)G.nslot * G.slot_bytes;
    // the launch is cooperative: every CTA must be resident at once
    int per_sm = 0;
    auto prepare = [&](auto kernel) {
        cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_limit);
        if (err == cudaSuccess) err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, c->threads, c->smem);
        return err;
    };
    if (tp) e = prepare(gemv_chain_kernel<512, 5, true>);
    else if (c->threads == 768) e = prepare(gemv_chain_kernel<768, 3, false>);
    else if (c->threads == 640) e = prepare(gemv_chain_kernel<640, 4, false>);
    else if (c->threads == 512) e = prepare(gemv_chain_kernel<512, 5, false>);
    else e = cudaErrorInvalidValue;
    if (e == cudaSuccess && per_sm < 1) e = cudaErrorLaunchOutOfResources;
    if (e == cudaSuccess) e = cudaMalloc(&c->d_ops, sizeof(ChainOp) * (size_t)n_ops);
    if (e == cudaSuccess && tp) c->d_counter = c->peers.counter[tp_rank];
    c->counter_bytes = 256 + (any_rescale ? 4 * (size_t)n_ops : 0);        // counters, then the largest |y| of every op
    c->counter_bytes = (size_t)round_up((int64_t)c->counter_bytes, 256);
    const size_t image_bytes = any_spread ? (size_t)G.nb_max * CHAIN_IMAGE_WORDS * 8 : 0;
    if (e == cudaSuccess && !tp) e = cudaMalloc(&c->d_counter, c->counter_bytes + image_bytes);
    if (e == cudaSuccess && any_spread && tp) e = cudaMalloc(&c->d_image, image_bytes);
    if (e == cudaSuccess && any_spread && tp && !zero_new_memory(c->d_image, image_bytes)) e = cudaErrorUnknown;      // no tag of any run
    if (e == cudaSuccess && any_spread && !tp) {
        c->d_image = reinterpret_cast<uint8_t *>(c->d_counter) + c->counter_bytes;
        c->counter_bytes += image_bytes;
    }
    if (e == cudaSuccess) e = cudaMemcpy(c->d_ops, rec.data(), sizeof(ChainOp) * (size_t)n_ops, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        bonsai_b200_chain_destroy(c);
        return (int)e;
    }
    *out = c;
    return 0;
}

int bonsai_b200_chain_create(const bonsai_b200_op *ops, int64_t n_ops, bonsai_b200_chain **out) {
    return chain_create_impl(ops, n_ops, 0, 1, nullptr, 0, 0, 0, out);
}

int bonsai_b200_chain_create_tp(const bonsai_b200_op *ops, int64_t n_ops, int rank, int world, const void *const *peer_base,
                                int64_t buffer_bytes, int64_t counter_offset, int64_t wait_limit_us,
                                bonsai_b200_chain **out) {
    if (world < 2) return 1;
    return chain_create_impl(ops, n_ops, rank, world, peer_base, buffer_bytes, counter_offset, wait_limit_us, out);
}

int bonsai_b200_chain_run(bonsai_b200_chain *c, bonsai_stream stream) {
    if (!c || !c->d_ops) return 1;
    cudaStream_t st = as_stream(stream);
    cudaError_t e = cudaSuccess;
    if (!c->tp) e = cudaMemsetAsync(c->d_counter, 0, c->counter_bytes > 256 ? c->counter_bytes : 2 * sizeof(unsigned int), st);      // and the image's tags
    if (e != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)c->grid);
    cfg.blockDim = dim3((unsigned)c->threads);
    cfg.dynamicSmemBytes = c->smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const ChainOp *ops = c->d_ops;
    auto go = [&](auto kernel) {
        return cudaLaunchKernelEx(&cfg, kernel, ops, c->n_ops, c->G, c->d_counter, c->d_image, c->peers);
    };
    if (c->tp) e = go(gemv_chain_kernel<512, 5, true>);
    else if (c->threads == 768) e = go(gemv_chain_kernel<768, 3, false>);
    else if (c->threads == 640) e = go(gemv_chain_kernel<640, 4, false>);
    else e = go(gemv_chain_kernel<512, 5, false>);
    return (int)e;
}

int bonsai_b200_chain_destroy(bonsai_b200_chain *c) {
    if (!c) return 0;
    cudaError_t e1 = c->d_ops ? cudaFree(c->d_ops) : cudaSuccess;
    cudaError_t e2 = (c->d_counter && !c->tp) ? cudaFree(c->d_counter) : cudaSuccess;
    if (c->d_image && c->tp) cudaFree(c->d_image);
    delete c;
    return (int)(e1 != cudaSuccess ? e1 : e2);
}

int bonsai_b200_chain_info(const bonsai_b200_chain *c, int64_t out[4]) {
    if (!c || !out) return 1;
    out[0] = c->threads;
    out[1] = c->G.nslot;
    out[2] = c->G.slot_bytes;
    out[3] = c->grid;
    return 0;
}

int bonsai_b200_gemv_chunk_sums(const void *W, const void *xq, int32_t *out, int64_t row0, int64_t n_rows,
                                int64_t n_in, bonsai_stream stream) {
    if (n_in <= 0 || n_in % 128 != 0 || row0 < 0) return 1;
    if (n_rows <= 0) return 0;
    if (n_rows > INT32_MAX || (reinterpret_cast<uintptr_t>(xq) & 3u)) return 1;
    const long long total = n_rows * (n_in / 32);
    long long blocks = (total + 255) / 256;
    if (blocks > 16 * SM_COUNT) blocks = 16 * SM_COUNT;
    gemv_chunk_sums_kernel<<<(unsigned)blocks, 256, 0, as_stream(stream)>>>(
        static_cast<const uint8_t *>(W), static_cast<const uint8_t *>(xq), out, row0, (int)n_rows, (int)(n_in / 128));
    return (int)cudaGetLastError();
}

int bonsai_b200_gemv_dump(const void *W, const void *xq, float *y, int32_t *sums, int64_t n_out, int64_t n_in,
                          bonsai_stream stream) {
    if (n_in <= 0 || n_in % 128 != 0 || n_out <= 0 || n_out > INT32_MAX || !sums) return 1;
    const int nblocks = (int)(n_in / 128);
    MmaGeom mp;
    int smem_bytes = 0, grid = 0;
    if (!aligned16(W) || !aligned4(xq) || !plan_mma(n_out, nblocks, 200, mp, smem_bytes, grid)) return 1;
    static SmemOptIn opt;
    cudaError_t err = opt.ensure(gemv_mma_kernel<true>);
    if (err != cudaSuccess) return (int)err;
    return (int)launch(gemv_mma_kernel<true>, dim3((unsigned)grid), dim3(MMA_THREADS), (size_t)smem_bytes, as_stream(stream),
                       false, static_cast<const uint8_t *>(W), static_cast<const uint32_t *>(xq), y, mp, sums);
}

// 2-D tensor map: dims {d0 (fastest), d1}, row stride in bytes, box {b0, b1}.  The encoder is a driver entry point; it is
// looked up through the runtime so that the library links against nothing but cudart.  false: not available (the
// caller takes a form that needs no map).
static bool tensor_map_2d(CUtensorMap *map, CUtensorMapDataType type, const void *base, uint64_t d0, uint64_t d1,
                          uint64_t stride_bytes, uint32_t b0, uint32_t b1, CUtensorMapSwizzle swizzle) {
    using Encode = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static Encode encode = [] {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            fn = nullptr;
        return reinterpret_cast<Encode>(fn);
    }();
    if (!encode) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)d0, (cuuint64_t)d1};
    const cuuint64_t strides[1] = {(cuuint64_t)stride_bytes};
    const cuuint32_t box[2] = {b0, b1};
    const cuuint32_t estr[2] = {1u, 1u};
    return encode(map, type, 2, const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// The two fp16 planes of the split activations, [2][n_tok][n_in]: box = 64 values x one tile of tokens x both planes, landing with
// the 128-byte swizzle the MMA reads; tokens past the end arrive as zeros.
static bool tensor_map_planes(CUtensorMap *map, const void *planes, uint64_t n_in, uint64_t n_tok, uint32_t tile_tokens) {
    using Encode = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !fn)
        return false;
    const cuuint64_t dims[3] = {n_in, n_tok, 2};
    const cuuint64_t strides[2] = {n_in * 2, n_tok * n_in * 2};
    const cuuint32_t box[3] = {64u, (cuuint32_t)tile_tokens, 2u};
    const cuuint32_t estr[3] = {1u, 1u, 1u};
    return reinterpret_cast<Encode>(fn)(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void *>(planes), dims, strides, box, estr,
                                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// A PQ2_0 matrix seen as [n_out][row_bytes / 4] 32-bit words, box = 68 words (8 blocks) x 128 rows.
static bool encode_w_map(CUtensorMap *map, const void *W, int64_t n_out, int64_t row_bytes) {
    return tensor_map_2d(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, W, (uint64_t)(row_bytes / 4), (uint64_t)n_out, (uint64_t)row_bytes,
                         68u, (uint32_t)TC_M, CU_TENSOR_MAP_SWIZZLE_NONE);
}

// Scratch of the fp16 tensor-core mat-mul: counts and two slots per CTA for its parts of tiles, the activations as two fp16 planes, a
// scale per token.  A call that gets none takes the integer kernel, which needs no scratch.
static constexpr size_t T16_COUNTS_BYTES = (size_t)T16_MAX_CTAS * T16_PART_COUNTS * sizeof(unsigned int);
static StreamScratch g_gemm_scratch(false);

// Scratch of the prompt attention: k and v as tile images, 2 KB per position and kv head, what k and v take themselves.  Prompts of one
// conversation grow a little each time.  A call that gets none takes the CUDA-core kernel.
static StreamScratch g_attn_scratch(true);

static std::atomic<unsigned int> g_gemm_epoch{0};       // launch number of the tensor-core mat-muls (tags partial-tile flags)

static void fill_tc_params(TcParams &P, int64_t n_out, int64_t n_in, int64_t n_tok, int tile_m, int tile_n) {
    P.n_out = (int)n_out;
    P.nblocks = (int)(n_in / 128);
    P.n_tok = (int)n_tok;
    P.tiles_tok = (int)((n_tok + tile_n - 1) / tile_n);
    P.n_tiles = (int)(((n_out + tile_m - 1) / tile_m) * P.tiles_tok);
    P.total_it = (long long)P.n_tiles * P.nblocks;
}

static constexpr size_t T16_PARTS_BYTES = (size_t)T16_MAX_CTAS * 2 * T16C<128, 2>::PART_FLOATS * sizeof(float);
static size_t tc16_scratch_bytes(int64_t n_in, int64_t n_tok) {
    return T16_COUNTS_BYTES + T16_PARTS_BYTES + 2 * (size_t)n_tok * (size_t)n_in * sizeof(__half) + (size_t)n_tok * sizeof(float);
}

// The fp16 tensor-core mat-mul (gemm_tc16.cuh).  -1: not taken (shape, alignment, no scratch, no tensor-map encoder).
extern "C++" {
static SmemOptIn g_tc16_pairs_smem;

// How a mat-mul is divided over `workers` CTAs (or pairs of them), and about how long that takes.
struct Tc16Plan {
    int tile_n = 0, grid = 0, stream_k = 0;
    long long tiles_tok = 0, tiles = 0;
    double ns = 0;
};
template <int TN, int CTAS>
static Tc16Plan plan_tc16(int64_t n_out, int64_t nblocks, int64_t n_tok, int workers) {
    Tc16Plan p;
    // As many token tiles as TN asks for, all of about the same width: the MMAs' time is the tokens' (37 tokens take 48 columns, not 64).
    const long long step = 16 * CTAS;
    p.tiles_tok = (n_tok + TN - 1) / TN;
    p.tile_n = (int)(((n_tok + p.tiles_tok - 1) / p.tiles_tok + step - 1) / step * step);
    p.tiles = (n_out + T16_M * CTAS - 1) / (T16_M * CTAS) * p.tiles_tok;
    if (p.tiles > INT32_MAX) return p;
    // Whole tiles in turn, or the blocks of all tiles in equal shares: at most four workers per tile on average (a tile that begins inside a share can
    // be cut into five parts), at least 16 blocks each.  Measured at
    // 33 - 192 tokens of 1024 -> 12288, 5120 -> 5120, 5120 -> 17408 and 17408 -> 5120: 5.5 us and 0.53 per block for a CTA, 8 us and 0.39 + 0.003 per token
    // and block for a pair, 7 us for leaving, fetching and adding the parts of tiles that are shared.
    const double start = CTAS == 1 ? 5500 : 8000, block = CTAS == 1 ? 530 : 390 + 3 * p.tile_n;
    const long long total = p.tiles * nblocks;
    p.grid = (int)std::min<long long>(p.tiles, workers);
    p.ns = start + block * (double)((p.tiles + workers - 1) / workers * nblocks);
    const long long sharing = p.tiles >= workers ? workers : std::min<long long>({total / 16, 4 * p.tiles, workers});
    if (p.tiles % workers != 0 && sharing >= p.grid && sharing > 1) {
        const double ns = start + block * (double)((total + sharing - 1) / sharing) + 7000;
        if (ns < p.ns) p.grid = (int)sharing, p.stream_k = 1, p.ns = ns;
    }
    return p;
}
static int tc16_workers(int ctas) {
    int dev = 0, sms = 0;
    if (ctas != 1) return std::min(g_tc16_pairs.ask(gemm_tc16_kernel<128, 2>, g_tc16_pairs_smem, 2, T16C<128, 2>::THREADS), T16_MAX_CTAS / ctas);
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    return std::min(sms, T16_MAX_CTAS);
}

// One launch over activations that lie in `planes`.
struct Tc16Args {
    float *Y;
    int64_t n_out, nblocks, n_tok;
    const float *scale;
    float *parts;
    unsigned int *counts;
    Tc16Maps maps;
};
template <int TN, int CTAS>
static cudaError_t launch_gemm_tc16_n(const Tc16Args &a, const Tc16Plan &plan, SmemOptIn &opt, cudaStream_t st) {
    T16Params P{};
    P.n_out = (int)a.n_out;
    P.nblocks = (int)a.nblocks;
    P.n_tok = (int)a.n_tok;
    P.tile_n = plan.tile_n;
    P.tiles_tok = (int)plan.tiles_tok;
    P.n_tiles = (int)plan.tiles;
    P.idesc = t16_idesc(plan.tile_n, CTAS);
    P.stream_k = plan.stream_k;
    P.per_worker = plan.tiles * a.nblocks / plan.grid;
    P.rest = (int)(plan.tiles * a.nblocks % plan.grid);
    cudaError_t e = opt.ensure(gemm_tc16_kernel<TN, CTAS>);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(plan.grid * CTAS));
    cfg.blockDim = dim3(T16C<TN, CTAS>::THREADS);
    cfg.dynamicSmemBytes = T16C<TN, CTAS>::SMEM_BYTES;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CTAS;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;        // behind the split, which does not write weights
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = CTAS == 1 ? attr + 1 : attr;
    cfg.numAttrs = (CTAS != 1) + (g_opt_overlap.load() != 0);
    if (CTAS != 1) return launch_clusters(cfg, gemm_tc16_kernel<TN, CTAS>, a.Y, P, a.scale, a.parts, a.counts, a.maps);
    return cudaLaunchKernelEx(&cfg, gemm_tc16_kernel<TN, CTAS>, a.Y, P, a.scale, a.parts, a.counts, a.maps);
}
}  // extern "C++"
// Tiles of up to 64 tokens by a CTA, or of up to 128 by a pair of CTAs (the code expansion is paid once per tile, and each CTA fetches half
// of the activations): what the plans say takes less time.  (us, a CTA / a pair: 64 tokens of 5120 -> 17408 26.8 / 30.8, 65 44.5 / 33.7, 129
// 61.7 / 59.6; of 5120 -> 5120, where pairs have too few tiles, 64 22.5 / 24.7, 128 25.3 / 29.0; 129 of 1024 -> 12288 20.6 / 22.9.)
static int launch_gemm_tc16(const void *W, const void *Xq, float *Y, int64_t n_out, int64_t n_in, int64_t n_tok, cudaStream_t st) {
    const int64_t nblocks = n_in / 128;
    if (nblocks % 8 != 0 || !aligned16(W) || !aligned4(Xq) || n_tok > (1 << 28)) return -1;
    const int tile = g_opt_gemm_tile.load(), sms = tc16_workers(1), pairs = tile != 64 && (n_tok > 64 || tile == 128) ? tc16_workers(2) : 0;
    if (sms <= 0) return -1;
    const Tc16Plan one = plan_tc16<64, 1>(n_out, nblocks, n_tok, sms);
    Tc16Plan two;
    if (pairs > 0) two = plan_tc16<128, 2>(n_out, nblocks, n_tok, pairs);
    const bool paired = pairs > 0 && two.tiles <= INT32_MAX && (tile == 128 || two.ns < one.ns);
    if (one.tiles > INT32_MAX) return -1;
    const size_t plane_bytes = (size_t)n_tok * (size_t)n_in * sizeof(__half);
    const StreamScratch::Lease lease = g_gemm_scratch.get(tc16_scratch_bytes(n_in, n_tok), st);      // held until the launches are enqueued
    uint8_t *ws = static_cast<uint8_t *>(lease.ptr);
    if (!ws) return -1;
    __half *planes = reinterpret_cast<__half *>(ws + T16_COUNTS_BYTES + T16_PARTS_BYTES);
    float *scale = reinterpret_cast<float *>(ws + T16_COUNTS_BYTES + T16_PARTS_BYTES + 2 * plane_bytes);
    alignas(64) Tc16Args a{Y, n_out, nblocks, n_tok, scale, reinterpret_cast<float *>(ws + T16_COUNTS_BYTES), reinterpret_cast<unsigned int *>(ws), {}};
    auto map_activations = [&](int tokens) { return tensor_map_planes(&a.maps.x, planes, (uint64_t)n_in, (uint64_t)n_tok, (uint32_t)tokens); };
    if (!encode_w_map(&a.maps.w, W, n_out, nblocks * W_BLOCK_BYTES) || !map_activations(paired ? two.tile_n / 2 : one.tile_n)) return -1;
    const int n_chunks = (int)(n_in / 32);
    const uint32_t *x32 = static_cast<const uint32_t *>(Xq);
    // slices: whole passes of a block, as many as bring about two blocks per SM
    const int groups = (int)((n_tok + 3) / 4);
    int passes = (n_chunks + T16_SPLIT_PASS - 1) / T16_SPLIT_PASS;
    passes = (int)((passes * groups + 2 * sms - 1) / (2 * sms));
    const int slice = passes * T16_SPLIT_PASS;
    const int counted = std::max(one.stream_k ? one.grid : 0, paired && two.stream_k ? 2 * two.grid : 0);      // CTAs that may count parts
    cudaError_t e = launch(groups <= 2 * sms ? tc16_split_kernel<true> : tc16_split_kernel<false>,
                           dim3((unsigned)groups, (unsigned)((n_chunks + slice - 1) / slice)), dim3(T16_SPLIT_THREADS), 0, st, true, x32, n_chunks, (int)n_tok, slice,
                           scale, planes, reinterpret_cast<uint4 *>(ws), counted * T16_PART_COUNTS / 4);
    if (e != cudaSuccess) return (int)e;
    if (paired) {
        e = launch_gemm_tc16_n<128, 2>(a, two, g_tc16_pairs_smem, st);
        if (!g_tc16_pairs.refused(e)) return (int)e;
        if (!map_activations(one.tile_n)) return -1;      // the same planes, by single CTAs: here, and in later calls from the start
    }
    static SmemOptIn opt;
    return (int)launch_gemm_tc16_n<64, 1>(a, one, opt, st);
}

// The tensor-core mat-mul: one CTA per SM walks its share of the (tile, weight block) iterations.
static int launch_gemm_tc(const void *W, const void *Xq, float *Y, int64_t n_out, int64_t n_in, int64_t n_tok,
                          int32_t *dump, cudaStream_t st) {
    TcParams P{};
    const long long tiles = (long long)((n_out + TC_M - 1) / TC_M) * ((n_tok + TC_N - 1) / TC_N);
    if (tiles > INT32_MAX) return 1;
    fill_tc_params(P, n_out, n_in, n_tok, TC_M, TC_N);
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return (int)e;
    if (sms > TC_MAX_CTAS - 1) sms = TC_MAX_CTAS - 1;
    const int grid = (int)(tiles < sms ? tiles : sms);
    // contiguous ranges when they are at least one tile long (then a tile is cut at most once); whole tiles otherwise
    P.stream_k = (tiles % grid != 0 && P.total_it / grid >= P.nblocks) ? 1 : 0;
    P.epoch = g_gemm_epoch.fetch_add(1) + 1u;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(TC_THREADS);
    cfg.dynamicSmemBytes = TC_SMEM_BYTES;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;        // a CTA may wait for its neighbour's partial tile: all must be resident
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const uint8_t *w8 = static_cast<const uint8_t *>(W);
    const uint32_t *x32 = static_cast<const uint32_t *>(Xq);
    // bulk-copy staging of the raw bytes needs 16-byte multiples everywhere; other shapes load from global memory
    alignas(64) CUtensorMap wmap;
    std::memset(&wmap, 0, sizeof(wmap));
    const bool tma = P.nblocks % 8 == 0 && n_tok % 4 == 0 && aligned16(W) && aligned16(Xq) &&
                     encode_w_map(&wmap, W, n_out, (int64_t)P.nblocks * W_BLOCK_BYTES);
    static SmemOptIn opt[4];
    auto go = [&](auto kernel, SmemOptIn &o, int smem) -> int {
        cudaError_t err = o.ensure(kernel);
        if (err != cudaSuccess) return (int)err;
        cfg.dynamicSmemBytes = (size_t)smem;
        return (int)cudaLaunchKernelEx(&cfg, kernel, w8, x32, Y, P, dump, wmap);
    };
    if (dump) return tma ? go(gemm_tc_kernel<true, true>, opt[0], TC_SMEM_BYTES_TMA) : go(gemm_tc_kernel<true, false>, opt[1], TC_SMEM_BYTES);
    return tma ? go(gemm_tc_kernel<false, true>, opt[2], TC_SMEM_BYTES_TMA) : go(gemm_tc_kernel<false, false>, opt[3], TC_SMEM_BYTES);
}

// The streaming small-batch mat-mul (gemv_mma.cuh).  -1: shape not taken (more than 8 tokens, odd block count, rows of
// more than 48 blocks that are not a multiple of 8 blocks, unaligned W, no tensor-map encoder in the driver).
static int launch_gemm_small(const void *W, const void *Xq, float *Y, int64_t n_out, int64_t n_in, int64_t n_tok,
                             int32_t *dump, cudaStream_t st) {
    if (n_tok < 1 || n_tok > 16 || (dump && n_tok > 8) || !aligned16(W) || n_out > INT32_MAX - 16) return -1;
    MmabGeom mp;
    int smem_bytes = 0, grid = 0;
    const int nb = (int)(n_in / 128);
    if (!plan_mmab(n_out, nb, (int)n_tok, 224, mp, smem_bytes, grid)) return -1;
    CUtensorMap wmap;
    std::memset(&wmap, 0, sizeof(wmap));
    if (mp.tiled && !tensor_map_2d(&wmap, CU_TENSOR_MAP_DATA_TYPE_UINT32, W, (uint64_t)nb * W_BLOCK_BYTES / 4, (uint64_t)n_out,
                                   (uint64_t)nb * W_BLOCK_BYTES, (uint32_t)(mp.stride / 4), 16u, CU_TENSOR_MAP_SWIZZLE_NONE))
        return -1;
    static SmemOptIn opt, opt2, opt_dump;
    mp.early = g_opt_pdl.load() != 0;
    if (mp.ntg == 2) {
        cudaError_t err = opt2.ensure(gemm_mma_kernel<false, 2, 1>);
        if (err != cudaSuccess) return (int)err;
        return (int)launch(gemm_mma_kernel<false, 2, 1>, dim3((unsigned)grid), dim3(MMAB_THREADS), (size_t)smem_bytes, st, true,
                           static_cast<const uint8_t *>(W), static_cast<const uint32_t *>(Xq), Y, mp, (int)n_tok, dump, wmap);
    }
    auto go = [&](auto kernel, SmemOptIn &o, bool with_pdl) -> int {
        cudaError_t err = o.ensure(kernel);
        if (err != cudaSuccess) return (int)err;
        return (int)launch(kernel, dim3((unsigned)grid), dim3(MMAB_THREADS), (size_t)smem_bytes, st, with_pdl,
                           static_cast<const uint8_t *>(W), static_cast<const uint32_t *>(Xq), Y, mp, (int)n_tok, dump, wmap);
    };
    static SmemOptIn opt_r2, opt_dump_r2;
    if (dump) return mp.nrg == 2 ? go(gemm_mma_kernel<true, 1, 2>, opt_dump_r2, false) : go(gemm_mma_kernel<true, 1, 1>, opt_dump, false);
    return mp.nrg == 2 ? go(gemm_mma_kernel<false, 1, 2>, opt_r2, true) : go(gemm_mma_kernel<false, 1, 1>, opt, true);
}

int bonsai_p40_gemm(const void *W, const void *Xq, float *Y, int64_t n_out, int64_t n_in, int64_t n_tok,
                    bonsai_stream stream) {
    if (n_in <= 0 || n_in % 128 != 0) return 1;
    if (n_out <= 0 || n_tok <= 0) return 0;
    if (n_out > INT32_MAX || n_tok > INT32_MAX || !aligned4(Xq)) return 1;
    const int path = g_opt_gemm_path.load();
    // One token is the mat-vec (chunk-major Xq of one token is the plain Q8_1 vector, Y[n_out][1] the output vector):
    // 8 us against 140 us of the integer SIMT kernel on 5120 -> 17408; same bits and options as bonsai_p40_gemv.
    if (n_tok == 1 && path < 0) return bonsai_p40_gemv(W, Xq, Y, n_out, n_in, stream);
    // From 9 tokens on the tensor cores win even with a 64-token tile mostly empty (5120 -> 17408 at 16 tokens:
    // 40 us against 140 us of the integer SIMT kernel); 2 .. 8 tokens stream the weights once through mma.sync.
    // 9 .. 16 tokens: the streaming kernel with two token groups per code extraction is ahead of the tensor cores
    // (31 against 40 us at 24 MB, 297 against 312 us at 338 MB); it needs rows of a multiple of 8 blocks.
    const bool small16 = n_tok >= 9 && n_tok <= 16 && (n_in / 128) % 8 == 0;
    if (path == 2 || (path < 0 && n_tok >= 2 && (n_tok <= 8 || small16))) {     // a handful of tokens: weights streamed once for all of them
        const int rc = launch_gemm_small(W, Xq, Y, n_out, n_in, n_tok, nullptr, as_stream(stream));
        if (rc >= 0) return rc;                                       // -1: the shape does not fit, a kernel below takes it
    }
    if (path == 1 || path == 3 || (path < 0 && n_tok >= 9)) {
        if (path != 3) {                                              // the fp16 form first; -1: it does not take the call
            const int rc = launch_gemm_tc16(W, Xq, Y, n_out, n_in, n_tok, as_stream(stream));
            if (rc >= 0) return rc;
        }
        return launch_gemm_tc(W, Xq, Y, n_out, n_in, n_tok, nullptr, as_stream(stream));
    }
    const dim3 grid((unsigned)((n_out + GS_ROWS - 1) / GS_ROWS), (unsigned)((n_tok + GS_TOKS - 1) / GS_TOKS));
    if (grid.y > 65535) return 1;
    gemm_simt_kernel<<<grid, 256, 0, as_stream(stream)>>>(static_cast<const uint8_t *>(W),
                                                          static_cast<const uint32_t *>(Xq), Y, (int)n_out,
                                                          (int)(n_in / 128), (int)n_tok);
    return (int)cudaGetLastError();
}

int bonsai_b200_gemm_release(void) {
    g_gemm_scratch.release();
    g_attn_scratch.release();
    return 0;
}

int bonsai_b200_gemm_reserve(int64_t n_in, int64_t n_tok, bonsai_stream stream) {
    if (n_in <= 0 || n_in % 128 != 0 || n_tok <= 0 || n_tok > (1 << 28)) return 1;
    return g_gemm_scratch.get(tc16_scratch_bytes(n_in, n_tok), as_stream(stream), true).ptr ? 0 : (int)cudaErrorMemoryAllocation;
}

int bonsai_b200_gemm_dump(const void *W, const void *Xq, float *Y, int32_t *sums, int64_t n_out, int64_t n_in,
                          int64_t n_tok, bonsai_stream stream) {
    if (n_in <= 0 || n_in % 128 != 0 || n_out <= 0 || n_tok <= 0 || !sums) return 1;
    if (n_out > INT32_MAX || n_tok > INT32_MAX || !aligned4(Xq)) return 1;
    if (n_tok <= 8) {           // the streaming small-batch kernel, when it takes the shape
        const int rc = launch_gemm_small(W, Xq, Y, n_out, n_in, n_tok, sums, as_stream(stream));
        if (rc >= 0) return rc;
    }
    return launch_gemm_tc(W, Xq, Y, n_out, n_in, n_tok, sums, as_stream(stream));
}

int bonsai_p40_repack(const void *src, void *dst, int64_t n_out, int64_t n_in, bonsai_stream stream) {
    if (n_in % 128 != 0 || n_out <= 0) return 1;
    const int64_t nb = n_in / 128;
    if (nb <= 0 || nb % 8 != 0 || nb > INT32_MAX / 64) return 1;
    if (!aligned16(dst) || (reinterpret_cast<uintptr_t>(src) & 1u)) return 1;
    const int64_t row_bytes = nb * W_BLOCK_BYTES;
    if (aligned16(src) && row_bytes <= RPK_SMEM_BYTES) {
        const int rows_per_pass = (int)(RPK_SMEM_BYTES / row_bytes);
        long long passes = (n_out + rows_per_pass - 1) / rows_per_pass;
        if (passes > 6 * SM_COUNT) passes = 6 * SM_COUNT;
        repack_staged_kernel<<<(unsigned)passes, 256, RPK_SMEM_BYTES, as_stream(stream)>>>(
            static_cast<const uint8_t *>(src), static_cast<uint8_t *>(dst), n_out, (int)nb, rows_per_pass);
        return (int)cudaGetLastError();
    }
    const long long total = n_out * 4 * nb;
    long long blocks = (total + 255) / 256;
    if (blocks > 32 * SM_COUNT) blocks = 32 * SM_COUNT;
    repack_kernel<<<(unsigned)blocks, 256, 0, as_stream(stream)>>>(static_cast<const uint8_t *>(src),
                                                                   static_cast<uint8_t *>(dst), n_out, (int)nb);
    return (int)cudaGetLastError();
}

int bonsai_p40_gemv_repack(const void *W, const float *x, float *y, int64_t n_out, int64_t n_in,
                           bonsai_stream stream) {
    if (n_in % 128 != 0 || n_out <= 0) return 1;
    const int64_t nb64 = n_in / 128;
    if (nb64 <= 0 || nb64 % 8 != 0 || n_out > INT32_MAX) return 1;
    const int nb = (int)nb64;
    const size_t row_bytes = (size_t)nb * W_BLOCK_BYTES;
    const size_t act_bytes = (size_t)4 * nb * RP_REC_WORDS * 4;
    // the reference refuses vectors whose Q8_1 image exceeds 48 KiB; this build takes anything that
    // leaves room for four rows beside the activation records
    if (GEMV_BAR_BYTES + act_bytes + 4 * row_bytes + 64 > (size_t)111 * 1024) return 1;
    if (!aligned16(W) || !aligned4(x)) return 1;        // dst of bonsai_p40_repack is 16-byte aligned; x is any float pointer
    const bool pdl = g_opt_pdl.load() != 0;
    GemvPlan p = plan_rows(n_out, row_bytes, act_bytes, 1, g_opt_gemv_variant.load());
    if (p.threads > 256) p.threads = 256;
    const dim3 grid((unsigned)p.ctas);
    static SmemOptIn opt[12];
    auto go = [&](auto kernel, SmemOptIn &o) -> cudaError_t {
        cudaError_t err = o.ensure(kernel);
        if (err != cudaSuccess) return err;
        return launch(kernel, grid, dim3(p.threads), (size_t)p.smem_bytes, as_stream(stream), pdl,
                      static_cast<const uint8_t *>(W), x, y, (int)n_out, nb, p.rows_per_cta, p.rows_per_stage);
    };
    // gemv_order 1: the terms of a row added in unit order by one lane (the bits of repack_row_dot); otherwise by a warp
    const bool tree = g_opt_gemv_order.load() != 1;
    const bool vec = aligned16(x);
    // the streaming kernel (ring of tiles, quantiser in the prologue) when it takes the shape: the default
    {
        StreamParams sp;
        int threads = 0, smem_bytes = 0;
        if (tree && vec && n_in % FWHT_N == 0 && plan_stream(n_out, nb, g_opt_gemv_variant.load(), sp, threads, smem_bytes)) {
            // Long rows: the CTAs of a cluster share the quantiser.  In fours where each of their CTAs finds an SM (clusters do not cross a group of
            // SMs: 147 CTAs in fours ran two to an SM in places and took twice as long), else in pairs, whose barrier is worth it from 96
            // blocks on.  us, alone / in pairs / in fours: 17408 -> 64 6.94 / 5.60 / 4.80, -> 1000 7.65 / 6.63 / 5.99, -> 5120 11.75 / 10.69 / 18.7;
            // 12288 -> 1056 6.14 / 6.05 / 5.19, -> 4096 8.49 / 8.37 / 14.8, -> 5120 9.04 / 8.97, -> 17408 17.97 / 17.77; 11264 -> 5120 8.42 / 8.45;
            // 5120 -> 64 3.55 / 3.55 / 3.18, -> 1056 3.96 / 4.16 / 3.81.  Fours with more than 28 rows per CTA are worth it from 80 blocks on: -> 4160,
            // alone / in fours and the same behind the rotation, 5120 4.54 / 5.13, 6.53 / 6.75; 9216 6.78 / 7.28, 8.79 / 8.80; 10240 7.38 / 7.37, 9.41 / 8.90.
            // (At 16 to 28 rows and 40 to 72 blocks fours are up to 7 % behind alone and up to 6 % ahead behind the rotation.)
            static SmemOptIn sopt[3];
            const unsigned ctas = (unsigned)((n_out + sp.rows_per_cta - 1) / sp.rows_per_cta);
            auto room = [&](ClusterRoom &r, auto kernel, SmemOptIn &o, unsigned cluster) { return ctas <= cluster * (unsigned)r.ask(kernel, o, cluster, 512); };
            unsigned cl = 1;
            if (nb >= (sp.rows_per_cta <= 28 ? 40 : 80) && room(g_repack_fours, gemv_stream_kernel<true, true, 4>, sopt[2], 4)) cl = 4;
            else if (nb >= 96 && room(g_repack_pairs, gemv_stream_kernel<true, true, 2>, sopt[1], 2)) cl = 2;
            sp.early = pdl;
            cudaLaunchAttribute attr[2];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
            attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[1].val.programmaticStreamSerializationAllowed = 1;
            cudaLaunchConfig_t cfg = {};
            cfg.blockDim = dim3(threads);
            cfg.dynamicSmemBytes = (size_t)smem_bytes;
            cfg.stream = as_stream(stream);
            auto go = [&](auto kernel, SmemOptIn &o) -> cudaError_t {
                cudaError_t err = o.ensure(kernel);
                if (err != cudaSuccess) return err;
                attr[0].val.clusterDim.x = cl;
                cfg.gridDim = dim3((ctas + cl - 1) / cl * cl);
                cfg.attrs = cl == 1 ? attr + 1 : attr;
                cfg.numAttrs = (cl > 1) + (g_opt_overlap.load() != 0);
                const uint8_t *w8 = static_cast<const uint8_t *>(W);
                const uint32_t *no_xq = nullptr;
                const float *no_signs = nullptr;
                uint32_t *no_out = nullptr;
                return cl > 1 ? launch_clusters(cfg, kernel, w8, no_xq, y, sp, x, no_signs, no_out) : cudaLaunchKernelEx(&cfg, kernel, w8, no_xq, y, sp, x, no_signs, no_out);
            };
            if (cl > 1) {
                const cudaError_t err = cl == 4 ? go(gemv_stream_kernel<true, true, 4>, sopt[2]) : go(gemv_stream_kernel<true, true, 2>, sopt[1]);
                if (!g_repack_fours.refused(err) || !g_repack_pairs.refused(err)) return (int)err;
                cl = 1;
            }
            return (int)go(gemv_stream_kernel<true, true>, sopt[0]);
        }
    }
    auto pick = [&](auto t, auto v, int base) -> cudaError_t {
        constexpr bool T = decltype(t)::value, V = decltype(v)::value;
        if (p.rr == 1) return go(gemv_repack_kernel<1, V, T>, opt[base]);
        if (p.rr == 2) return go(gemv_repack_kernel<2, V, T>, opt[base + 1]);
        return go(gemv_repack_kernel<4, V, T>, opt[base + 2]);
    };
    cudaError_t e;
    if (tree) e = vec ? pick(std::true_type{}, std::true_type{}, 0) : pick(std::true_type{}, std::false_type{}, 3);
    else e = vec ? pick(std::false_type{}, std::true_type{}, 6) : pick(std::false_type{}, std::false_type{}, 9);
    return (int)e;
}

int bonsai_b200_ptq1_pack(const void *src, void *dst, int64_t n_blocks, uint64_t *code3_count, bonsai_stream stream) {
    if (n_blocks <= 0) return n_blocks == 0 ? 0 : 1;
    if ((reinterpret_cast<uintptr_t>(src) & 1u) || (reinterpret_cast<uintptr_t>(dst) & 1u) || !code3_count ||
        (reinterpret_cast<uintptr_t>(code3_count) & 7u))
        return 1;
    long long blocks = (n_blocks + 255) / 256;
    if (blocks > 16 * SM_COUNT) blocks = 16 * SM_COUNT;
    ptq1_pack_kernel<<<(unsigned)blocks, 256, 0, as_stream(stream)>>>(static_cast<const uint8_t *>(src), static_cast<uint8_t *>(dst),
                                                                      n_blocks, reinterpret_cast<unsigned long long *>(code3_count));
    return (int)cudaGetLastError();
}

int bonsai_b200_ptq1_unpack(const void *src, void *dst, int64_t n_blocks, bonsai_stream stream) {
    if (n_blocks <= 0) return n_blocks == 0 ? 0 : 1;
    if ((reinterpret_cast<uintptr_t>(src) & 1u) || (reinterpret_cast<uintptr_t>(dst) & 1u)) return 1;
    long long blocks = (n_blocks + 255) / 256;
    if (blocks > 16 * SM_COUNT) blocks = 16 * SM_COUNT;
    ptq1_unpack_kernel<<<(unsigned)blocks, 256, 0, as_stream(stream)>>>(static_cast<const uint8_t *>(src), static_cast<uint8_t *>(dst),
                                                                        n_blocks);
    return (int)cudaGetLastError();
}

int bonsai_b200_synth_pq2_0(void *W, int64_t first_block, int64_t n_blocks, uint64_t seed, bonsai_stream stream) {
    if (n_blocks <= 0) return n_blocks == 0 ? 0 : 1;
    if (reinterpret_cast<uintptr_t>(W) & 1u) return 1;
    long long blocks = (n_blocks * 17 + 255) / 256;
    if (blocks > 64 * SM_COUNT) blocks = 64 * SM_COUNT;
    synth_pq2_kernel<<<(unsigned)blocks, 256, 0, as_stream(stream)>>>(static_cast<unsigned short *>(W), first_block,
                                                                      n_blocks, seed);
    return (int)cudaGetLastError();
}

int bonsai_b200_stream_probe(const void *buf, int64_t bytes, int mode, void *sink, bonsai_stream stream) {
    if (bytes <= 0 || !aligned16(buf) || !sink) return 1;
    if (mode == 0) {
        probe_ldg_kernel<<<SM_COUNT * 8, 256, 0, as_stream(stream)>>>(static_cast<const uint4 *>(buf), bytes / 16,
                                                                     static_cast<unsigned *>(sink));
    } else if (mode == 1) {
        const int slot = 16384, stages = 6;
        if (bytes < slot) return 1;
        static SmemOptIn opt;
        cudaError_t e = opt.ensure(probe_bulk_kernel);
        if (e != cudaSuccess) return (int)e;
        probe_bulk_kernel<<<SM_COUNT * 2, 32, 128 + slot * stages, as_stream(stream)>>>(
            static_cast<const uint8_t *>(buf), bytes, slot, stages, static_cast<unsigned *>(sink));
    } else {
        return 1;
    }
    return (int)cudaGetLastError();
}

int bonsai_b200_set_option(const char *key, int64_t value) {
    if (!key) return 1;
    if (!std::strcmp(key, "pdl")) { g_opt_pdl.store(value != 0); return 0; }
    if (!std::strcmp(key, "overlap")) { g_opt_overlap.store(value != 0); return 0; }
    if (!std::strcmp(key, "gemv_order")) {
        if (value < 0 || value > 2) return 1;
        g_opt_gemv_order.store((int)value);
        return 0;
    }
    if (!std::strcmp(key, "gemm_path")) { g_opt_gemm_path.store((int)value); return 0; }
    if (!std::strcmp(key, "fuse_linear")) { g_opt_fuse_linear.store(value < 0 ? -1 : value != 0); return 0; }
#ifdef BONSAI_B200_TUNING
    // Geometry knobs of the test build (build.py --tuning, the default of this repository's build script): they let the
    // parity tests force every tiling.  A build without the macro has no such keys and always uses the tuned defaults.
    if (!std::strcmp(key, "gemv_variant")) { g_opt_gemv_variant.store((int)value); return 0; }
    if (!std::strcmp(key, "chain_threads")) {
        if (value != 512 && value != 640 && value != 768) return 1;
        g_opt_chain_threads.store((int)value);
        return 0;
    }
    if (!std::strcmp(key, "chain_seg")) {
        if (value < 8 || value > 8 * STREAM_STEPS || value % 8 != 0) return 1;
        g_opt_chain_seg.store((int)value);
        return 0;
    }
    if (!std::strcmp(key, "chain_spread_nb")) {
        if (value < 0) return 1;
        g_opt_chain_spread_nb.store((int)value);
        return 0;
    }
    if (!std::strcmp(key, "gemm_tile")) {
        if (value != 0 && value != 64 && value != 128) return 1;
        g_opt_gemm_tile.store((int)value);
        return 0;
    }
    if (!std::strcmp(key, "refuse_clusters")) {         // 0 forgets the refusals too
        if (value < 0) return 1;
        g_opt_refuse_clusters.store((int)value);
        if (value == 0) {
            g_tc16_pairs.forget(), g_repack_pairs.forget(), g_repack_fours.forget();
            for (auto &few : g_few_clusters) few.forget();
        }
        return 0;
    }
    if (!std::strcmp(key, "kv_wide")) { g_opt_kv_wide.store(value != 0); return 0; }
    if (!std::strcmp(key, "kv_push")) { g_opt_kv_push.store(value != 0); return 0; }
    if (!std::strcmp(key, "chain_tile_kb")) {
        if (value < 4 || value > 48) return 1;
        g_opt_chain_tile_kb.store((int)value);
        return 0;
    }
#endif
    return 1;
}

int bonsai_b200_device_status(void) {
    int v = -1;
    cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess) return (int)e + 1000;
    e = cudaMemcpyFromSymbol(&v, g_device_status, sizeof(int));
    if (e != cudaSuccess) return (int)e + 1000;
    return v;
}

int bonsai_b200_clear_status(void) {
    const int zero = 0;
    cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess) return (int)e + 1000;
    e = cudaMemcpyToSymbol(g_device_status, &zero, sizeof(int));
    return e == cudaSuccess ? 0 : (int)e + 1000;
}

int bonsai_b200_version(void) { return 200; }

// ---- the operators beside the mat-vec path (reference: include/bonsai_p40.h:44-56) ---------------------------
int bonsai_p40_rmsnorm(const float *x, const float *w, float *y, int64_t n_rows, int64_t n, float eps,
                       bonsai_stream stream) {
    // return convention of src/kernels/elementwise_p40.cu:82-88
    if (n <= 0 || n_rows <= 0) return (n <= 0) ? 1 : 0;
    if (n > INT32_MAX || n_rows > INT32_MAX || !aligned4(x) || !aligned4(w) || !aligned4(y)) return 1;
    const bool vec = n % 4 == 0 && aligned16(x) && aligned16(w) && aligned16(y);
    const dim3 threads(32 * (unsigned)std::min<int64_t>(RMS_WARPS, (n + 127) / 128));
    // Behind one row comes its projection, which asks for its weights in front of its wait: it is let in at once.  Behind rows comes a batch's quantiser, which has nothing
    // to ask for: let in by ending.  us by ending / at once: one row with bonsai_b200_linear 1024 -> 4096 (replayed by a graph) 4.35 / 3.95, 5120 -> 64 5.69 / 5.40, -> 1024 6.72 / 6.22,
    // -> 1850 7.12 / 6.38, 8192 -> 600 7.76 / 7.22; rows with quantiser and mat-mul 12 x 1024 7.72 / 7.98, 8 x 5120 -> 17408 18.57 / 18.66, -> 5120 13.37 / 13.24, 37 x 5120 23.16 / 23.18,
    // 100 x 6144 31.9 / 33.1, 148 x 3072 23.1 / 25.6, x 5120 30.8 / 35.0.
    const bool early = n_rows == 1;
    auto run = [&](auto kernel) {
        return (int)launch(kernel, dim3((unsigned)n_rows), threads, 0, as_stream(stream), true, x, w, y, (int)n, eps);
    };
    auto go = [&](auto hold) {
        constexpr int HOLD = decltype(hold)::value;
        if (early) return vec ? run(rmsnorm_kernel<true, HOLD, true>) : run(rmsnorm_kernel<false, HOLD, true>);
        return vec ? run(rmsnorm_kernel<true, HOLD, false>) : run(rmsnorm_kernel<false, HOLD, false>);
    };
    // Rows that fit stay in registers, which costs CTAs per SM: with 16-byte accesses and up to five slices per warp that is ahead at any
    // count of rows (5120 values, 8192 rows: 54 us, 70 us read twice), with eight up to four rows per SM (6144 values, 512 rows: 5.8 and 7.0 us,
    // 2048 rows: 24 and 20), with scalar accesses up to three (5120 values, 400 rows: 6.4 and 6.9 us, 1024 rows: 12.5 and 10.1).
    if (n_rows <= (vec ? 4 : 3) * SM_COUNT || (vec && n <= 5 * 1024)) {
        if (n <= 1024) return go(std::integral_constant<int, 1>{});
        if (n <= 2 * 1024) return go(std::integral_constant<int, 2>{});
        if (n <= 3 * 1024) return go(std::integral_constant<int, 3>{});
        if (n <= 5 * 1024 && vec) return early ? run(rmsnorm_kernel<true, 5, true>) : run(rmsnorm_kernel<true, 5, false>);
        if (n <= 8 * 1024) return go(std::integral_constant<int, 8>{});
    }
    if (!vec && n_rows > 2 * SM_COUNT) return run(rmsnorm_kernel<false, -1, false>);
    return go(std::integral_constant<int, 0>{});
}

int bonsai_b200_swiglu(const float *gate, const float *up, float *y, int64_t n, bonsai_stream stream) {
    if (n <= 0 || n > INT32_MAX || !aligned4(gate) || !aligned4(up) || !aligned4(y)) return 1;
    const bool vec = n % 4 == 0 && aligned16(gate) && aligned16(up) && aligned16(y);
    const int64_t threads = vec ? n / 4 : n;
    const int64_t ctas = (threads + 255) / 256;
    auto run = [&](auto kernel) { return (int)launch(kernel, dim3((unsigned)ctas), dim3(256), 0, as_stream(stream), true, gate, up, y, (int)n); };
    // us, the next launch let in by ending / at once: 5120 values with bonsai_b200_linear -> 1024 6.17 / 5.64; with quantiser and mat-mul 8 x 5120 12.8 / 12.6, 16 x 5120 13.0 /
    // 12.9, 8 x 17408 (136 CTAs) 23.2 / 23.1, 12 x 17408 39.2 / 39.5, 64 x 17408 41.1 / 44.8.
    if (ctas <= SM_COUNT) return vec ? run(swiglu_kernel<true, true>) : run(swiglu_kernel<false, true>);
    return vec ? run(swiglu_kernel<true, false>) : run(swiglu_kernel<false, false>);
}

int bonsai_p40_gdn_step(float *state, const float *q, const float *k, const float *v, const float *g, const float *beta,
                        float *out, int n_k_heads, int n_v_heads, int K, int V, bonsai_stream stream) {
    // rejections of src/kernels/attn_p40.cu:121-124
    if (V <= 0 || V % 32 != 0 || K <= 0 || K > GDN_KMAX) return 1;
    if (n_v_heads <= 0 || n_k_heads <= 0 || n_v_heads % n_k_heads != 0) return 1;
    const int blocks = n_v_heads * (V / 32);
    return (int)launch(gdn_step_kernel, dim3((unsigned)blocks), dim3(GDN_WARPS * 32), 0, as_stream(stream), true, state, q, k, v, g, beta, out, n_k_heads,
                       n_v_heads, K, V);
}

static size_t attn_scratch_bytes(int n_tok, int n_head_kv) { return (size_t)((n_tok + ATC_KEYS - 1) / ATC_KEYS) * n_head_kv * ATC_IMG_BYTES; }

// Attention on the tensor cores (attn_tc.cuh).  -1: not taken (no scratch to be had).
static int launch_attn_tc(const float *q, const float *k, const float *v, float *out, int n_tok, int n_head, int n_head_kv, float scale, cudaStream_t st) {
    const int tiles = (n_tok + ATC_KEYS - 1) / ATC_KEYS;
    const long long ctas = (long long)n_head * ((n_tok + ATC_M - 1) / ATC_M);
    if (ctas > INT32_MAX || n_head_kv > 65535) return -1;
    const StreamScratch::Lease lease = g_attn_scratch.get(attn_scratch_bytes(n_tok, n_head_kv), st);      // held until both launches are enqueued
    uint8_t *images = static_cast<uint8_t *>(lease.ptr);
    if (!images) return -1;
    static SmemOptIn opt;
    cudaError_t e = opt.ensure(attn_tc_kernel);
    if (e == cudaSuccess)
        e = launch(attn_planes_kernel, dim3((unsigned)tiles, (unsigned)n_head_kv, 2), dim3(ATC_PREP_THREADS), 0, st, true, k, v, images, n_tok, n_head_kv);
    if (e == cudaSuccess)
        e = launch(attn_tc_kernel, dim3((unsigned)ctas), dim3(ATC_THREADS), (size_t)ATC_SMEM_BYTES, st, true, q, k, v, images, out, n_tok, n_head, n_head_kv, scale);
    return (int)e;
}

int bonsai_b200_attn_reserve(int n_tok, int n_head_kv, bonsai_stream stream) {
    if (n_tok <= 0 || n_head_kv <= 0) return 1;
    if (n_tok < ATC_MIN_TOKENS || n_head_kv > 65535) return 0;          // served without scratch
    return g_attn_scratch.get(attn_scratch_bytes(n_tok, n_head_kv), as_stream(stream), true).ptr ? 0 : (int)cudaErrorMemoryAllocation;
}

int bonsai_p40_attn(const float *q, const float *k, const float *v, float *out, int n_tok, int n_head, int n_head_kv,
                    int head_dim, float scale, bonsai_stream stream) {
    // rejections of src/kernels/attn_p40.cu:134-136
    if (head_dim != ATT_D || n_head_kv == 0 || (n_head % n_head_kv) != 0) return 1;
    if (n_tok <= 0 || n_head <= 0 || n_head_kv <= 0) return (n_tok <= 0) ? 0 : 1;
    if (!aligned16(k) || !aligned16(v) || !aligned4(q) || !aligned4(out)) return 1;    // rows of 256 floats: 16-byte loads
    if ((long long)n_head * ((n_tok + 31) / 32) > INT32_MAX) return 1;
    if (n_tok >= ATC_MIN_TOKENS) {
        const int rc = launch_attn_tc(q, k, v, out, n_tok, n_head, n_head_kv, scale, as_stream(stream));
        if (rc >= 0) return rc;
    }
    // CTAs of 16 queries, or of 8 where those of 16 fill only half of the SMs or leave the last of two or three rounds half empty.  us by 16, 8 queries: 24 heads,
    // 16 tokens 6.5 / 4.9, 30 7.9 / 7.0, 70 12.6 / 13.2, 100 18.4 / 20.1, 130 26.3 / 26.8, 150 33.9 / 31.1, 191 49.2 / 37.4; 64 heads, 50 15.8 / 12.4, 100 31.5 / 25.6 (a fourth round
    // of four CTAs: not looked for), 160 47.9 / 52.5, 191 60.8 / 72.6.  (Of 32 queries, with eight warps: 16 tokens 6.4, 191 45.3; 64 heads 191 76.)
    static SmemOptIn opt[2];
    const long long of16 = (long long)n_head * ((n_tok + 15) / 16);
    const bool few = 2 * of16 <= SM_COUNT || (2 * of16 > 3 * SM_COUNT && of16 <= 3 * SM_COUNT);
    const int warps = few ? 2 : 4;
    auto kernel = few ? attn_kernel<2> : attn_kernel<4>;
    cudaError_t err = opt[few].ensure(kernel);
    if (err != cudaSuccess) return (int)err;
    const long long ctas = (long long)n_head * ((n_tok + warps * ATT_QPW - 1) / (warps * ATT_QPW));
    if (ctas > INT32_MAX) return 1;
    return (int)launch(kernel, dim3((unsigned)ctas), dim3((unsigned)(32 * warps)), (size_t)att_smem_bytes(warps), as_stream(stream), true, q, k, v, out, n_tok, n_head, n_head_kv, scale);
}

// ---- K/V cache (reference: include/bonsai_kv.h, src/kernels/kv_p40.cu:247-367) ----------------------------------
// Geometry of the 27B model (include/bonsai_model.h:29-52): 16 full-attention layers, 24 query / 4 kv heads of 256;
// 48 linear-attention layers with 48 value heads of 128 x 128 state.
namespace {
constexpr int KVM_FULL = 16, KVM_HEADS = 24, KVM_KV_HEADS = 4, KVM_CONTEXT = 262144;
constexpr int KVM_LINEAR = 48, KVM_V_HEADS = 48, KVM_STATE = 128;
constexpr int KV_SPLIT_MIN = 2 * KV_TILE;      // positions
constexpr int KVM_GROUP = KVM_HEADS / KVM_KV_HEADS;
inline int64_t kv_array_bytes(int capacity) { return (int64_t)KVM_FULL * KVM_KV_HEADS * capacity * KV_ROW; }
inline int64_t kv_gdn_bytes() { return (int64_t)KVM_LINEAR * KVM_V_HEADS * KVM_STATE * KVM_STATE * (int64_t)sizeof(float); }
constexpr int KV_COUNTERS = KVM_KV_HEADS * KV_CLUSTER;      // per layer
inline size_t kv_ws_floats(int max_clusters) { return (size_t)KVM_KV_HEADS * KV_CLUSTER * max_clusters * KV_REC; }      // per layer

// The decode kernel in clusters of 8 (or, wide, of 16) CTAs.  push: tile buffers of the form for one cluster per kv head, 0 the form for several.
using KvKernel = decltype(&kv_attn_kernel<KVM_GROUP>);
inline KvKernel kv_kernel(bool wide, int push) {
    static const KvKernel kernels[2][3] = {{kv_attn_kernel<KVM_GROUP, KV_CLUSTER, 0>, kv_attn_kernel<KVM_GROUP, KV_CLUSTER, 1>, kv_attn_kernel<KVM_GROUP, KV_CLUSTER, 2>},
                                           {nullptr, kv_attn_kernel<KVM_GROUP, KV_WIDE_CLUSTER, 1>, kv_attn_kernel<KVM_GROUP, KV_WIDE_CLUSTER, 2>}};
    return kernels[wide][push];
}
inline unsigned kv_threads(int push) { return push ? 32 * KV_PUSH_WARPS : KV_THREADS; }
inline unsigned kv_smem(int push) { return push ? KV_PUSH_SMEM_BYTES + push * 2 * KV_HALF_BYTES : KV_SMEM_BYTES; }
// Its clusters that are resident at once on the current device (0: they do not run here).  Asked once per device.
int kv_resident(bool wide, int push) {
    static std::atomic<int> known[2][3][64];
    static SmemOptIn opt[2][3];
    int dev = 0, resident = 0;
    const KvKernel kernel = kv_kernel(wide, push);
    if (opt[wide][push].ensure(kernel) != cudaSuccess || cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (dev < 64 && (resident = known[wide][push][dev].load(std::memory_order_relaxed)) > 0) return resident;
    if (wide && cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    const unsigned cluster = wide ? KV_WIDE_CLUSTER : KV_CLUSTER;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cluster * KV_MAX_CLUSTERS, KVM_KV_HEADS);
    cfg.blockDim = dim3(kv_threads(push));
    cfg.dynamicSmemBytes = kv_smem(push);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&resident, kernel, &cfg) != cudaSuccess || resident <= 0) {
        (void)cudaGetLastError();
        return 0;
    }
    if (dev < 64) known[wide][push][dev].store(resident, std::memory_order_relaxed);
    return resident;
}
// Clusters of eight per kv head that a device with so many of them resident gets at most: one wave.
inline int kv_max_clusters(int resident) { return resident <= 0 ? 0 : std::min(std::max(resident / KVM_KV_HEADS, 1), KV_MAX_CLUSTERS); }

// How n_pos positions of a kv head are divided: clusters of `cluster` CTAs, a split per CTA, `chunk` positions per split.
struct KvSplits {
    int cluster, clusters, chunk;
};
KvSplits kv_splits(int n_pos, int max_clusters, bool wide_runs) {
    // One cluster (eight splits) per kv head until a split has KV_SPLIT_MIN positions -- two tiles, both in flight at once --
    // then more, up to what is resident at once (one wave).  Splits are multiples of 16 positions (a warp's share of a
    // tile), not of whole tiles: at 32 768 positions the longest is 5 % longer than the mean instead of 12 %.
    KvSplits s{KV_CLUSTER, std::max(1, std::min(n_pos / (KV_CLUSTER * KV_SPLIT_MIN), max_clusters)), 0};
    // One cluster of 16 where one or two of eight would do and each of their splits would have more than a tile, 513 to 3071 positions: 701
    // are a tile a split, not two one after the other, and 2048 need no merge through memory.  16 layers with their appends, in us,
    // with clusters of 8 and of 16 (both merged by reading): 513 positions 145 / 126, 701 148 / 128, 1501 180 / 150, 2048 187 / 158, 3001 213 / 186.  Up to 512 a split
    // of eight is one tile already (401 positions 102 by eight, 103 by 16; 271 102 and 101); from 3072 on three clusters of eight have more splits than the one of 16 that the kernel is laid out for.
    if (wide_runs && n_pos > KV_CLUSTER * KV_TILE && n_pos < 3 * KV_CLUSTER * KV_SPLIT_MIN) s.cluster = KV_WIDE_CLUSTER, s.clusters = 1;
    const int n_split = s.cluster * s.clusters;
    s.chunk = (((n_pos + n_split - 1) / n_split) + 15) / 16 * 16;
    return s;
}
// Clusters of 16 serve where those of all kv heads run at once; in waves they would be slower than clusters of eight.
inline bool kv_wide_runs(int resident_wide) { return g_opt_kv_wide.load() && resident_wide >= KVM_KV_HEADS; }
}  // namespace

struct bonsai_kv_cache {
    int capacity = 0;
    uint8_t *d_k = nullptr, *d_v = nullptr;
    float *d_gdn = nullptr, *d_ws = nullptr;
    unsigned int *d_counters = nullptr;         // behind the workspace's records; records and counters are a layer's own, so
                                                // that layers may be decoded on different streams at once
    int max_clusters = 1;                       // clusters of eight of the decode kernel per kv head, at most
    int resident_wide = 0;                      // clusters of 16 that are resident at once
    bool push_runs = false;                     // whether the form for one cluster of eight per kv head runs here
};

int64_t bonsai_kv_bytes(int capacity) {
    if (capacity <= 0) return 0;
    if (capacity > KVM_CONTEXT) capacity = KVM_CONTEXT;
    return 2 * kv_array_bytes(capacity);
}
int64_t bonsai_kv_gdn_bytes(void) { return kv_gdn_bytes(); }

bonsai_kv_cache *bonsai_kv_create(int capacity, bonsai_stream stream) {
    if (capacity <= 0) return nullptr;
    if (capacity > KVM_CONTEXT) capacity = KVM_CONTEXT;
    bonsai_kv_cache *kv = new (std::nothrow) bonsai_kv_cache;
    if (!kv) return nullptr;
    kv->capacity = capacity;
    kv->max_clusters = kv_max_clusters(kv_resident(false, 0));
    kv->resident_wide = std::min(kv_resident(true, 1), kv_resident(true, 2));
    kv->push_runs = std::min(kv_resident(false, 1), kv_resident(false, 2)) > 0;
    const size_t ws = (size_t)KVM_FULL * kv_ws_floats(kv->max_clusters) * sizeof(float), ncnt = (size_t)KVM_FULL * KV_COUNTERS * sizeof(unsigned int);
    if (kv->max_clusters <= 0 || cudaMalloc(&kv->d_k, (size_t)kv_array_bytes(capacity)) != cudaSuccess ||
        cudaMalloc(&kv->d_v, (size_t)kv_array_bytes(capacity)) != cudaSuccess || cudaMalloc(&kv->d_gdn, (size_t)kv_gdn_bytes()) != cudaSuccess ||
        cudaMalloc(&kv->d_ws, ws + ncnt) != cudaSuccess) {
        bonsai_kv_free(kv);
        return nullptr;
    }
    kv->d_counters = reinterpret_cast<unsigned int *>(reinterpret_cast<char *>(kv->d_ws) + ws);
    // the counters are zero before the first launch on any stream, and the caller's stream is not waited for
    if (!zero_new_memory(kv->d_counters, ncnt)) {
        bonsai_kv_free(kv);
        return nullptr;
    }
    (void)cudaMemsetAsync(kv->d_gdn, 0, (size_t)kv_gdn_bytes(), as_stream(stream));
    return kv;
}

void bonsai_kv_free(bonsai_kv_cache *kv) {
    if (!kv) return;
    cudaFree(kv->d_k);
    cudaFree(kv->d_v);
    cudaFree(kv->d_gdn);
    cudaFree(kv->d_ws);
    delete kv;
}

void bonsai_kv_reset(bonsai_kv_cache *kv, bonsai_stream stream) {
    if (kv) (void)cudaMemsetAsync(kv->d_gdn, 0, (size_t)kv_gdn_bytes(), as_stream(stream));
}

float *bonsai_kv_gdn_state(bonsai_kv_cache *kv, int layer) {
    if (!kv || layer < 0 || layer >= KVM_LINEAR) return nullptr;
    return kv->d_gdn + (size_t)layer * KVM_V_HEADS * KVM_STATE * KVM_STATE;
}

int bonsai_kv_append_batch(bonsai_kv_cache *kv, int layer, int pos0, int n_tok, const float *k, const float *v,
                           bonsai_stream stream) {
    if (!kv || !k || !v) return 1;
    if (layer < 0 || layer >= KVM_FULL) return 1;
    if (n_tok <= 0 || pos0 < 0 || (long long)pos0 + n_tok > kv->capacity) return 1;
    const int nrow = n_tok * KVM_KV_HEADS;
    // any float pointer is taken; 16-byte aligned ones get 16-byte loads
    const bool vec = aligned16(k) && aligned16(v);
    const int blocks = (nrow + KV_APPEND_WARPS - 1) / KV_APPEND_WARPS;
    const bool early = blocks <= 8 * SM_COUNT;              // 2368 tokens: one wave of eight blocks of 256 threads per SM
    auto kernel = early ? (vec ? kv_append_kernel<true, true> : kv_append_kernel<false, true>)
                        : (vec ? kv_append_kernel<true, false> : kv_append_kernel<false, false>);
    return (int)launch(kernel, dim3((unsigned)blocks), dim3(32 * KV_APPEND_WARPS), 0, as_stream(stream), true, kv->d_k, kv->d_v, k, v, pos0, n_tok,
                       KVM_KV_HEADS, kv->capacity, layer);
}

int bonsai_kv_append(bonsai_kv_cache *kv, int layer, int pos, const float *k, const float *v, bonsai_stream stream) {
    return bonsai_kv_append_batch(kv, layer, pos, 1, k, v, stream);
}

int bonsai_kv_attn_decode(bonsai_kv_cache *kv, int layer, int pos, const float *q, float *out, bonsai_stream stream) {
    if (!kv || !q || !out) return 1;
    if (layer < 0 || layer >= KVM_FULL) return 1;
    if (pos < 0 || pos >= kv->capacity) return 1;
    const KvSplits s = kv_splits(pos + 1, kv->max_clusters, kv_wide_runs(kv->resident_wide));
    const bool wide = s.cluster == KV_WIDE_CLUSTER;
    const int push = s.clusters == 1 && (wide || (kv->push_runs && g_opt_kv_push.load())) ? (s.chunk <= KV_TILE ? 1 : 2) : 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(s.cluster * s.clusters), KVM_KV_HEADS);
    cfg.blockDim = dim3(kv_threads(push));
    cfg.dynamicSmemBytes = kv_smem(push);
    cfg.stream = as_stream(stream);
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)s.cluster;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g_opt_overlap.load() ? 2 : 1;
    return (int)cudaLaunchKernelEx(&cfg, kv_kernel(wide, push), q, (const uint8_t *)kv->d_k, (const uint8_t *)kv->d_v,
                                   kv->d_ws + (size_t)layer * kv_ws_floats(kv->max_clusters), kv->d_counters + layer * KV_COUNTERS, out,
                                   pos, s.chunk, KVM_KV_HEADS, kv->capacity, layer, 0.0625f);
}

int bonsai_b200_kv_splits(int n_pos, int resident8, int resident16, int64_t out[3]) {
    if (n_pos <= 0 || n_pos > KVM_CONTEXT || !out) return 1;
    const int max_clusters = kv_max_clusters(resident8 < 0 ? kv_resident(false, 0) : resident8);
    if (max_clusters <= 0) return 1;
    const KvSplits s = kv_splits(n_pos, max_clusters, kv_wide_runs(resident16 < 0 ? std::min(kv_resident(true, 1), kv_resident(true, 2)) : resident16));
    out[0] = s.cluster;
    out[1] = s.clusters;
    out[2] = s.chunk;
    return 0;
}

// Test access to the cache arrays (byte parity of the quantiser): device pointers of K and V.
int bonsai_b200_kv_arrays(bonsai_kv_cache *kv, void **k, void **v, int64_t *bytes_each) {
    if (!kv || !k || !v || !bytes_each) return 1;
    *k = kv->d_k;
    *v = kv->d_v;
    *bytes_each = kv_array_bytes(kv->capacity);
    return 0;
}

}  // extern "C"
