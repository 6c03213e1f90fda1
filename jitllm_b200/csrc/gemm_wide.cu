// Quantised matrix-matrix product for more than 128 rows of activations (prompt chunks, wide stand-alone
// products): Y[n][rows] = X[n][cols] . W[rows][cols]^T on CTA pairs, same operands as gemm_tc.cu (weights rounded
// once to binary16 by the same code, activations as binary16 hi + lo parts, binary32 accumulation).
//
// What bounds it: the tensor pipe (ncu: 73 % active in the 8B gate/up launch of 512 rows, issue slots 41 %), the rest the
// start and the reading out of tiles, which nothing hides. A tile is 256 weight rows on two SMs (cta_group::2, M = 256):
// each CTA converts its own 128 rows into its own tensor memory and stages one half of the tokens, which both tensor cores
// read. Against 128 tokens converting a stage takes about as long as multiplying by it.
//
// The tensor core cuts every addition off at the accumulator's last place. Lo products (2^-11 of the hi ones) added into the
// hi sum lose those bits and cut it off twice as often: side by side in one accumulator of 256 tokens, a product of 4096
// columns was 9.2e-6 from the 64-bit sum (2-norm, weights that binary16 holds exactly); 4.4e-6 is what the hi sum alone
// costs, here and in gemm_tc.cu. Two forms keep to that:
//   * 192 tokens, an accumulator for either part (384 of the 512 tensor-memory columns) and four operand stages of 64 K
//     elements in the rest;
//   * 256 tokens, one accumulator, and a pair walks its part of the tile twice, first against the lo parts, then against the
//     hi parts: it converts twice, but reads out and hands over once.
// The second is taken where it has one tile to the first's two, for 193 to 256 rows. 14336 x 4096 Q4_K (device time of a
// stand-alone product, cold L2) in the first / the second form: 256 rows 81 / 69 us, 300 83 / 104, 384 85 / 108, 512 113 /
// 112, 2048 362 / 388. Tiles of 128 or 160 tokens are no faster than those of 192 (300 rows: 107 / 83 / 82 us).
//
// One persistent CTA pair per two SMs; the work list (256-row tile, token tile, 256-column raw stage) is cut into equal
// ranges, one per pair, as in gemm_tc.cu. Roles in a CTA, meeting only at mbarriers:
//   * warps 0-7: epilogue. They read the accumulator, add the residual and write Y (or a partial tile where a range
//     ends inside a tile; the pair that arrives last at the tile adds the others' partials to its accumulator, in pair
//     order). The conversion warps help with the last tile of a range.
//   * warps 8-19: convert raw units of 64 columns and store them into tensor memory. They never wait for the
//     epilogue, so the next tile's operands are ready when the accumulator is free.
//   * warp 20 of the pair's first CTA: issues the MMAs of both.
//   * warp 21: raw weight stages by TMA; warp 22: this CTA's half of the activation rows by TMA, completing on the
//     first CTA's barrier.
// Every wait is bounded; a wait that runs out sets the status word and the CTA winds down.
//
// Measured against the 64-token kernel, which converted weights and activations again for every tile, the splitting of the
// activations included: 14336 x 4096 against 512 rows Q4_K 263 -> 114 us, Q8_0 269 -> 118; against 129 rows 116 -> 54, 300
// rows 175 -> 83, 2048 rows 982 -> 370; Q8_0 4096 x 4096 against 512 rows 98 -> 54. The partial tiles folded out of memory
// alone, by the epilogue's warps, took 15-19 us of a launch; keeping the last arriver's share in tensor memory and lending
// it the idle conversion warps brought a 4096 x 4096 product from 55 to 41 us (when both parts shared an accumulator).
#include "gemm_tc_core.cuh"

#include <cstring>

namespace jl {
namespace {

constexpr int kPairM = 256;   // weight rows per tile, 128 per CTA
constexpr int kUnitK = 64;    // columns per operand stage: one unit per row, one 128-byte swizzle row per token
constexpr int kEpiWarps = 8, kConvWarps = 12;
constexpr int kConvGroups = kConvWarps / 4;  // a group of four warps converts one operand stage (128 rows)
constexpr int kWideThreads = (kEpiWarps + kConvWarps + 3) * 32;
constexpr uint32_t kAStageCols = kUnitK / 2, kWideTmemCols = 512;
constexpr int kMaxN = 256;    // most tokens per tile

// The two forms: NT tokens per tile, half of them staged per CTA.
template <int NT>
struct WideForm {
    static_assert(NT == 192 || NT == 256, "see the head of this file");
    static constexpr int passes = NT == 192 ? 1 : 2;
    static constexpr int acc_cols = passes == 1 ? 2 * NT : NT;  // an accumulator for either part of the activations, or one
    static constexpr int b_part = NT / 2 * kUnitK * 2;           // bytes: the hi or the lo part of a CTA's tokens
    static constexpr int b_stage = passes == 1 ? 2 * b_part : b_part;
    // Stages of the weights, in the tensor-memory columns that the accumulators leave, and of the activations: as many of
    // either, a stage's hand-back frees both.
    static constexpr int stages = passes == 1 ? 4 : 6;
    static_assert(acc_cols + stages * int(kAStageCols) <= int(kWideTmemCols), "tensor memory");
};

template <int TYPE, int NT>
struct WideSmem {
    static constexpr int bar_bytes = 512;
    static constexpr int b_bytes = WideForm<NT>::stages * WideForm<NT>::b_stage;
    static constexpr int raw_stage = RawFmt<TYPE>::stage_bytes;
    static constexpr int raw_fit = (227 * 1024 - 1024 - bar_bytes - b_bytes) / raw_stage;
    static constexpr int raw_stages = raw_fit > 4 ? 4 : raw_fit;
    static constexpr int raw_off = b_bytes;
    static constexpr int bar_off = raw_off + raw_stages * raw_stage;
    static constexpr int total = bar_off + bar_bytes + 1024;
    static_assert(raw_stages >= 2 && total <= 227 * 1024, "shared memory budget");
};

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The address of a barrier of the pair's first CTA, in the cluster window.
__device__ __forceinline__ uint32_t leader_addr(uint32_t smem_addr) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(smem_addr));
    return a;
}
// An arrival on a barrier of the other CTA. What it announces lies in tensor memory (stored and waited for, or read out,
// with the tcgen05 fence in front), never in memory that the other CTA reads with ordinary loads, so the default
// semantics are enough: a release at cluster scope costs a memory barrier per arrival.
__device__ __forceinline__ void arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// A bounded wait without a sleep between polls, for the one warp that issues the MMAs.
__device__ __forceinline__ bool wait_pair(uint32_t bar, uint32_t parity, uint32_t limit = (1u << 25)) {
    for (uint32_t i = 0; i < limit; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok != 0) return true;
    }
    return false;
}
// A word at the same place in the shared memory of either CTA of the pair (rank 0 or 1).
__device__ __forceinline__ void store_in_cta(uint32_t smem_addr, uint32_t rank, uint32_t value) {
    asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %0, %1;\n\tst.shared::cluster.u32 [a], %2;\n\t}" ::"r"(smem_addr),
                 "r"(rank), "r"(value)
                 : "memory");
}
// One activation box into this CTA's shared memory, completing on a barrier of the pair's first CTA.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t leader_bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(leader_bar)
        : "memory");
}
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred pe;\n\t.reg .b16 mask;\n\t"
        "elect.sync _|pe, 0xffffffff;\n\t"
        "mov.b16 mask, 3;\n\t"
        "@pe tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], mask;\n\t}"
        ::"r"(bar) : "memory");
}
// One MMA, by one elected lane of a converged warp.
__device__ __forceinline__ void umma_pair(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t b_hi, uint32_t idesc,
                                          uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred pe, pacc;\n\t.reg .b64 bd;\n\t"
        "elect.sync _|pe, 0xffffffff;\n\t"
        "setp.ne.b32 pacc, %5, 0;\n\t"
        "mov.b64 bd, {%2, %3};\n\t"
        "@pe tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], bd, %4, pacc;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate)
        : "memory");
}
// The MMAs of one operand stage (four K = 16 steps; one pass: against the hi part of the activations and, into the accumulator
// beside it, against the lo part) and the commit that hands the stage back to both CTAs.
template <int NT>
__device__ __forceinline__ void umma_stage_pair(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t b_hi, uint32_t done_bar,
                                                uint32_t accumulate_first) {
    using F = WideForm<NT>;
    // D fp32, A and B fp16, both K-major, M = 256, N = NT
    constexpr uint32_t idesc = (1u << 4) | (uint32_t(NT >> 3) << 17) | (uint32_t(kPairM >> 4) << 24);
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
        umma_pair(d_tmem, a_tmem + 8u * k, b_lo + 2u * k, b_hi, idesc, k == 0 ? accumulate_first : 1u);
        if (F::passes == 1)
            umma_pair(d_tmem + NT, a_tmem + 8u * k, b_lo + uint32_t(F::b_part >> 4) + 2u * k, b_hi, idesc, k == 0 ? accumulate_first : 1u);
    }
    umma_commit_pair(done_bar);
}
// The last of the stages 0 .. issued - 1 that went through slot s of a ring, or -1.
constexpr __host__ __device__ int last_in_slot(int issued, int s, int slots) {
    return issued > s ? issued - 1 - (issued - 1 - s) % slots : -1;
}
static_assert(last_in_slot(0, 0, 8) == -1 && last_in_slot(5, 5, 8) == -1 && last_in_slot(6, 5, 8) == 5, "first round");
static_assert(last_in_slot(8, 7, 8) == 7 && last_in_slot(9, 0, 8) == 8 && last_in_slot(9, 1, 8) == 1, "second round");

// Waits in the pair's first CTA for the activation boxes of both that a launch which gave up has left on their way: issued0
// and issued1 of the CTAs' stages. They complete on this CTA's barriers, a phase per stage, so the latest phase of a slot is
// armed for what will still arrive there: both boxes, or the one CTA's if the other has stopped a round earlier.
__device__ __forceinline__ void drain_activations(uint64_t *b_full, int slots, uint32_t stage_bytes, int issued0, int issued1) {
    for (int s = 0; s < slots; ++s) {
        const int last0 = last_in_slot(issued0, s, slots), last1 = last_in_slot(issued1, s, slots);
        const int last = last0 > last1 ? last0 : last1;
        if (last < 0) continue;
        if (last0 < last) mbar_expect_tx(b_full + s, stage_bytes);
        if (last1 < last)
            asm volatile("mbarrier.complete_tx.relaxed.cluster.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b_full + s)), "r"(stage_bytes)
                         : "memory");
        mbar_poll_bounded(b_full + s, uint32_t(last / slots) & 1u);
    }
}

// Where a pair's share of a tile goes and what is added to it on the way.
struct TileOut {
    float *y;          // first token, this thread's row
    const float *res;  // same place in the residual, or NULL
    float *slot;       // this CTA's partial slot, this thread's row
    int rows, ntok;
    bool inside;       // the row exists
};

// The tensor-memory instructions below are .sync.aligned: the whole warp executes each of them together. Whatever may have
// split it (a lane's arrival, a poll that lanes leave at different times, a row past the matrix) is followed by a
// __syncwarp() or a vote before the next one.

// 16 columns of this pair's sum. One pass: hi sum + lo sum, whose accumulator lies NT columns after the other's; its columns
// come eight at a time (what a finished tile also needs fills the registers).
template <int NT>
__device__ __forceinline__ void load_sum(uint32_t acc, int c0, float (&v)[16]) {
    __syncwarp();
    tmem_ld16(acc + uint32_t(c0), v);
    if constexpr (WideForm<NT>::passes == 1) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            uint32_t lo[8];
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                         : "=r"(lo[0]), "=r"(lo[1]), "=r"(lo[2]), "=r"(lo[3]), "=r"(lo[4]), "=r"(lo[5]), "=r"(lo[6]), "=r"(lo[7])
                         : "r"(acc + uint32_t(NT + c0 + 8 * h)));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int j = 0; j < 8; ++j) v[8 * h + j] += __uint_as_float(lo[j]);
        }
    }
}

// This CTA's partial tile into its slot: 16-column groups g0, g0 + step, ... of the accumulator.
template <int NT>
__device__ __forceinline__ void store_partial(const TileOut &o, uint32_t acc, int g0, int step) {
#pragma unroll 1
    for (int c0 = g0 * 16; c0 < o.ntok; c0 += step * 16) {
        float v[16];
        load_sum<NT>(acc, c0, v);
#pragma unroll
        for (int j = 0; j < 16; ++j) o.slot[size_t(c0 + j) * kTileM] = v[j];
    }
}

// The finished tile: the accumulator, the other pairs' partial tiles in pair order around it, the residual. own: this
// pair's place among the contributors c_first .. c_last (equal if there is one). A warp handles 16 columns at a time, a
// row per lane, so every load and store is 128 contiguous bytes; all loads of one source are in flight together, and the
// residual's are issued before the accumulator is read.
template <int NT>
__device__ __forceinline__ void finish_tile(const GemmArgs &a, const TileOut &o, uint32_t acc, int g0, int step, int c_first,
                                            int c_last, int own, uint32_t rank, int rr) {
    constexpr size_t slot_floats = size_t(kTileM) * kMaxN;
#pragma unroll 1
    for (int c0 = g0 * 16; c0 < o.ntok; c0 += step * 16) {
        float v[16], sum[16], res[16];
        if (o.res != nullptr && o.inside) {
#pragma unroll
            for (int j = 0; j < 16; ++j) res[j] = c0 + j < o.ntok ? o.res[size_t(c0 + j) * o.rows] : 0.f;
        }
#pragma unroll 1
        for (int c = c_first; c <= c_last; ++c) {
            if (c == own) {
                load_sum<NT>(acc, c0, v);
            } else {
                // only the first contributor's range starts before the tile
                const float *slot = a.scratch + (size_t(c * 2 + int(rank)) * 2 + (c == c_first ? 1 : 0)) * slot_floats + rr;
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = __ldcg(slot + size_t(c0 + j) * kTileM);
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) sum[j] = c == c_first ? v[j] : sum[j] + v[j];
        }
        if (o.inside) {
            if (o.res != nullptr) {
#pragma unroll
                for (int j = 0; j < 16; ++j) sum[j] = res[j] + sum[j];
            }
#pragma unroll
            for (int j = 0; j < 16; ++j)
                if (c0 + j < o.ntok) o.y[size_t(c0 + j) * o.rows] = sum[j];
        }
    }
}

template <int TYPE, int NT>
__global__ void __launch_bounds__(kWideThreads, 1)
    gemm_wide_kernel(const GemmArgs a, const __grid_constant__ CUtensorMap tm0, const __grid_constant__ CUtensorMap tm1,
                     const __grid_constant__ CUtensorMap tm2, const __grid_constant__ CUtensorMap tmx) {
    extern __shared__ uint8_t smem_raw[];
    using S = WideSmem<TYPE, NT>;
    using F = WideForm<NT>;
    using R = RawFmt<TYPE>;
    constexpr int RS = S::raw_stages, AS = F::stages;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t rank = cluster_rank();
    // 1024-byte aligned base (the swizzle pattern is a function of the shared address); the same in both CTAs.
    uint8_t *base = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t *bars = reinterpret_cast<uint64_t *>(base + S::bar_off);
    uint64_t *a_full = bars;               // [AS] first CTA: operand stage converted by both CTAs
    uint64_t *done = a_full + AS;          // [AS] the stage's MMAs are complete (both CTAs)
    uint64_t *b_full = done + AS;          // [AS] first CTA: both halves of the activation rows landed
    uint64_t *raw_full = b_full + AS;      // [RS]
    uint64_t *raw_empty = raw_full + RS;   // [RS]
    uint64_t *acc_full = raw_empty + RS;   // accumulator finished (both CTAs)
    uint64_t *acc_empty = acc_full + 1;    // first CTA: accumulator read out by both CTAs
    uint64_t *epi_bar = acc_empty + 1;     // the epilogue warps' own barrier
    uint64_t *last_fold = epi_bar + 1;     // it is known whether the range's last tile is finished here
    static_assert((3 * AS + 2 * 4 + 4) * 8 + 96 <= S::bar_bytes, "barrier block");
    uint32_t *tmem_ptr = reinterpret_cast<uint32_t *>(base + S::bar_off + S::bar_bytes - 16);
    volatile uint32_t *fold_flags = reinterpret_cast<uint32_t *>(base + S::bar_off + S::bar_bytes - 64);  // four, taken in turn
    volatile uint32_t *last_flags = fold_flags - 4;
    volatile uint32_t *abort_flag = tmem_ptr + 2;
    // The same in both CTAs at the end: the activation stages that either has issued, and whether either gave up.
    volatile uint32_t *pair_issued = last_flags - 4, *pair_abort = pair_issued + 2;

    int tiles = 0;
    for (int s = 0; s < a.nseg; ++s) tiles += (a.seg[s].rows + kPairM - 1) / kPairM;
    const int n_tiles = (a.n + NT - 1) / NT;
    const int raw_total = a.cols / kRawK;  // the second pass over them is not counted
    const int total = tiles * n_tiles * raw_total;
    const int pairs = int(gridDim.x >> 1), pair = int(blockIdx.x >> 1);
    const int lo = range_lo(total, pair, pairs), hi = range_lo(total, pair + 1, pairs);

    if (warp == kEpiWarps + kConvWarps) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_ptr)),
                     "r"(kWideTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int s = 0; s < AS; ++s) {
            mbar_init(a_full + s, 2 * 4);  // four warps of each CTA convert a stage
            mbar_init(done + s, 1);
            mbar_init(b_full + s, 1);
        }
        for (int s = 0; s < RS; ++s) {
            mbar_init(raw_full + s, 1);
            mbar_init(raw_empty + s, 4 * 4);  // four units, four warps each
        }
        mbar_init(acc_full, 1);
        mbar_init(acc_empty, 2 * kEpiWarps);
        mbar_init(epi_bar, kEpiWarps);
        mbar_init(last_fold, 1);
        mbar_fence_init();
        *abort_flag = 0u;
        pair_abort[0] = pair_abort[1] = 0u;
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // the pair's barriers exist and its tensor memory is allocated
    tc_fence_after();
    const uint32_t tmem_d = *tmem_ptr;
    pdl_launch_dependents();

    const auto locate = [&](int tile) {
        TileRef t = {0, 0};
        for (int s = 0; s < a.nseg; ++s) {
            const int of = (a.seg[s].rows + kPairM - 1) / kPairM;
            if (tile < of || s == a.nseg - 1) {
                t.seg = s;
                t.row0 = tile * kPairM + int(rank) * kTileM;
                break;
            }
            tile -= of;
        }
        return t;
    };
    const int lane_grp = warp & 3;  // epilogue: tensor-memory lanes 32 * lane_grp ..
    const auto tile_out = [&](int u, int which) {
        const TileRef tr = locate(u / n_tiles);
        const int tok0 = (u % n_tiles) * NT, rr = lane_grp * 32 + lane, row = tr.row0 + rr;
        const GemmSeg &seg = a.seg[tr.seg];
        const size_t at = size_t(tok0) * seg.rows + row;
        TileOut o;
        o.y = seg.y + at;
        o.res = seg.res != nullptr ? seg.res + at : nullptr;
        o.slot = a.scratch + (size_t(blockIdx.x) * 2 + which) * (size_t(kTileM) * kMaxN) + rr;
        o.rows = seg.rows;
        o.ntok = min(NT, a.n - tok0);
        o.inside = row < seg.rows;
        return o;
    };
    bool ok = true;

    if (warp == kEpiWarps + kConvWarps + 1) {
        // ---- raw weight stages, once a pass: this CTA's 128 rows (past the end of the matrix: zeros) ------
        if (lane == 0) {
            const uint64_t policy = policy_evict_first();
            fence_proxy_async();
            int i = 0;
            for (int f = lo, seg_end; f < hi && ok && *abort_flag == 0u; f = seg_end) {
                const int u = f / raw_total;
                seg_end = min((u + 1) * raw_total, hi);
                const TileRef tr = locate(u / n_tiles);
                const CUtensorMap *tmap = tr.seg == 0 ? &tm0 : (tr.seg == 1 ? &tm1 : &tm2);
                const int len = seg_end - f;
                for (int k = 0; k < F::passes * len && *abort_flag == 0u; ++k, ++i) {
                    const int r = f + (k < len ? k : k - len) - u * raw_total;
                    const int st = i % RS;
                    if (i >= RS && !(ok = mbar_poll_bounded(raw_empty + st, uint32_t(i / RS - 1) & 1u))) break;
                    mbar_expect_tx(raw_full + st, R::stage_bytes);
                    if (n_tiles == 1 && k >= (F::passes - 1) * len)  // read for the last time; otherwise the next reader finds the stage in L2
                        tma_load_2d(base + S::raw_off + st * R::stage_bytes, tmap, r * (R::row_bytes / 4), tr.row0, raw_full + st,
                                    policy);
                    else
                        tma_load_2d_plain(base + S::raw_off + st * R::stage_bytes, tmap, r * (R::row_bytes / 4), tr.row0,
                                          raw_full + st);
                }
            }
            // no copy may still be on its way into this CTA (after a wait that ran out: nobody may have read them)
            for (int k = i > RS ? i - RS : 0; k < i; ++k) mbar_poll_bounded(raw_full + k % RS, uint32_t(k / RS) & 1u);
        }
    } else if (warp == kEpiWarps + kConvWarps + 2) {
        // ---- activation rows: this CTA's half of the tile's tokens; two passes: the lo parts, then the hi parts
        if (lane == 0) {
            pdl_wait();
            const int stages = (hi - lo) * 4 * F::passes;
            int q = 0, s = 0;
            uint32_t par = 1;  // of the hand-back before the last round's
            for (int f = lo, seg_end; f < hi && ok && *abort_flag == 0u; f = seg_end) {
                const int u = f / raw_total;
                seg_end = min((u + 1) * raw_total, hi);
                const int tok = (u % n_tiles) * NT + int(rank) * (NT / 2), k_lo = (f - u * raw_total) * kRawK;
                const int len = 4 * (seg_end - f);
                for (int k = 0; k < F::passes * len && *abort_flag == 0u; ++k, ++q) {
                    if (q >= AS && !(ok = mbar_poll_bounded(done + s, par))) break;
                    if (rank == 0) mbar_expect_tx(b_full + s, 2 * F::b_stage);
                    const uint32_t dst = smem_u32(base) + uint32_t(s * F::b_stage), bar = leader_addr(smem_u32(b_full + s));
                    const int k0 = k_lo + (k < len ? k : k - len) * kUnitK;
                    tma_load_2d_pair(dst, &tmx, k0, (F::passes == 2 && k < len ? a.x_lo_row : 0) + tok, bar);
                    if (F::passes == 1) tma_load_2d_pair(dst + F::b_part, &tmx, k0, a.x_lo_row + tok, bar);
                    if (++s == AS) {
                        s = 0;
                        par ^= 1u;
                    }
                }
            }
            for (uint32_t r = 0; r < 2; ++r) store_in_cta(smem_u32(const_cast<uint32_t *>(pair_issued + rank)), r, uint32_t(q));
            // every hand-back has arrived here before this CTA may leave
            if (*abort_flag == 0u)
                for (int k = stages > AS ? stages - AS : 0; k < stages && ok; ++k)
                    ok = mbar_poll_bounded(done + k % AS, uint32_t(k / AS) & 1u);
        }
    } else if (warp == kEpiWarps + kConvWarps) {
        // ---- tensor-core issue (first CTA of the pair) -----------------------------------------------------
        if (rank == 0) {
            const uint32_t b_lo0 = sw128_desc_lo(smem_u32(base));
            const uint32_t a_full0 = smem_u32(a_full), done0 = smem_u32(done), b_full0 = smem_u32(b_full);
            int st = 0, turn = 0, issued = 0;
            uint32_t par = 0;
            int f = lo;
            while (f < hi && ok && *abort_flag == 0u) {
                const int u_hi = (f / raw_total + 1) * raw_total;
                const int seg_end = u_hi < hi ? u_hi : hi;
                const int nstage = 4 * F::passes * (seg_end - f);
                if (turn > 0) ok = __all_sync(0xffffffffu, wait_pair(smem_u32(acc_empty), uint32_t(turn - 1) & 1u));
                for (int k = 0; k < nstage && ok; ++k) {
                    ok = wait_pair(a_full0 + 8u * uint32_t(st), par) && wait_pair(b_full0 + 8u * uint32_t(st), par);
                    if (!__all_sync(0xffffffffu, ok)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    umma_stage_pair<NT>(tmem_d, tmem_d + uint32_t(F::acc_cols) + uint32_t(st) * kAStageCols,
                                        b_lo0 + uint32_t(st) * uint32_t(F::b_stage >> 4), kSw128DescHi, done0 + 8u * uint32_t(st),
                                        k == 0 ? 0u : 1u);
                    ++issued;
                    if (++st == AS) {
                        st = 0;
                        par ^= 1u;
                    }
                }
                if (!__all_sync(0xffffffffu, ok)) {
                    ok = false;
                    break;
                }
                umma_commit_pair(smem_u32(acc_full));
                ++turn;
                f = seg_end;
            }
            // the MMAs are over before the tensor memory is given back, whatever ended the loop
            if (issued > 0) wait_pair(done0 + 8u * uint32_t((issued - 1) % AS), uint32_t((issued - 1) / AS) & 1u);
            __syncwarp();
        }
    } else if (warp >= kEpiWarps) {
        // ---- conversion: groups of four warps take the units in turn --------------------------------------
        const int grp = (warp - kEpiWarps) >> 2, row = lane_grp * 32 + lane;
        const uint32_t raw_row0 = smem_u32(base + S::raw_off) + uint32_t(row) * R::row_bytes;
        const uint32_t tm_col0 = tmem_d + (uint32_t(row & ~31) << 16) + uint32_t(F::acc_cols);
        const uint32_t raw_full0 = smem_u32(raw_full), raw_empty0 = smem_u32(raw_empty), done0 = smem_u32(done);
        const uint32_t a_full_lead = leader_addr(smem_u32(a_full));
        int pending = -1;
        // A stage is published one stage late: its tensor-memory stores have landed by the time the next unit is converted.
        const auto publish = [&]() {
            if (pending < 0) return;
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) arrive_cluster(a_full_lead + 8u * uint32_t(pending));
            __syncwarp();
            pending = -1;
        };
        int s = grp, rev = 0, st = 0, unit = grp;
        uint32_t raw_par = 0;
        static_assert(kConvGroups <= 4 && kConvGroups <= AS, "running indices advance by less than a raw stage");
        const int stages = (hi - lo) * 4 * F::passes;
        for (int q = grp; q < stages && *abort_flag == 0u; q += kConvGroups) {
            ok = mbar_poll_bounded_u32(raw_full0 + 8u * uint32_t(st), raw_par);
            if (!__all_sync(0xffffffffu, ok)) {
                ok = false;
                break;
            }
            UnitRegs<TYPE> unit_regs;
            unit_load<TYPE>(raw_row0 + uint32_t(st) * uint32_t(R::stage_bytes), unit, unit_regs);
            uint32_t cols[16];
            unit_convert<TYPE>(unit_regs, 0, cols);
            // Published ahead of the wait for this stage's columns: where the accumulators leave four operand stages, that wait
            // lasts until the stage before the published one has been multiplied.
            publish();
            if (rev > 0) ok = mbar_poll_bounded_u32(done0 + 8u * uint32_t(s), uint32_t(rev - 1) & 1u);
            if (!__all_sync(0xffffffffu, ok)) {
                ok = false;
                break;
            }
            tc_fence_after();
            const uint32_t col0 = tm_col0 + uint32_t(s) * kAStageCols;
            tmem_st16(col0, cols);
            unit_convert<TYPE>(unit_regs, 1, cols);
            tmem_st16(col0 + 16u, cols);
            pending = s;
            __syncwarp();
            if (lane == 0) mbar_arrive_u32(raw_empty0 + 8u * uint32_t(st));
            s += kConvGroups;
            if (s >= AS) {
                s -= AS;
                ++rev;
            }
            unit += kConvGroups;
            if (unit >= 4) {
                unit -= 4;
                if (++st == RS) {
                    st = 0;
                    raw_par ^= 1u;
                }
            }
        }
        __syncwarp();
        if (ok)
            publish();
        else
            tmem_wait_st();  // no store may be on its way when the tensor memory is given back
        // The range's last tile, if this pair finishes it: these warps are idle by then.
        if (ok) ok = __all_sync(0xffffffffu, mbar_poll_bounded(last_fold, 0u));
        if (ok && last_flags[0] != 0u) {
            const int u = (hi - 1) / raw_total;
            tc_fence_after();
            __threadfence();
            finish_tile<NT>(a, tile_out(u, 0), tmem_d + (uint32_t(lane_grp * 32) << 16), warp >> 2, (kEpiWarps + kConvWarps) / 4,
                        int(last_flags[1]), int(last_flags[2]), pair, rank, lane_grp * 32 + lane);
        }
    } else {
        // ---- epilogue -----------------------------------------------------------------------------------
        pdl_wait();  // results, residuals and the partial-tile workspace belong to the kernel ahead until here
        const int col_grp = warp >> 2;
        const uint32_t acc = tmem_d + (uint32_t(lane_grp * 32) << 16);
        const uint32_t acc_empty_lead = leader_addr(smem_u32(acc_empty));
        int turn = 0, epi_phase = 0, flag_turn = 0;
        const auto epi_sync = [&]() {
            __syncwarp();
            if (lane == 0) mbar_arrive(epi_bar);
            const bool there = mbar_poll_bounded(epi_bar, uint32_t(epi_phase) & 1u);
            ++epi_phase;
            return bool(__all_sync(0xffffffffu, there));
        };
        int f = lo;
        while (f < hi && *abort_flag == 0u) {
            const int u = f / raw_total, u_lo = u * raw_total;
            const int seg_end = u_lo + raw_total < hi ? u_lo + raw_total : hi;
            const bool whole = f == u_lo && seg_end == u_lo + raw_total, last = seg_end == hi;
            // partial slot: 0 if this pair's range starts inside the tile, 1 if it only ends inside it
            const TileOut o = tile_out(u, f > u_lo ? 0 : 1);
            int c_first = pair, c_last = pair;
            if (!whole) {
                c_first = cta_of(total, u_lo, pairs);
                c_last = cta_of(total, u_lo + raw_total - 1, pairs);
            }
            ok = mbar_poll_bounded(acc_full, uint32_t(turn) & 1u);
            if (!__all_sync(0xffffffffu, ok)) {
                ok = false;
                break;
            }
            ++turn;
            tc_fence_after();
            bool mine = whole;  // this pair writes the result
            if (!whole) {
                // The pair that comes last finishes the tile from its accumulator. If the others have all arrived there
                // is no partial to store (the usual case: the ranges on both sides of a cut end at different times);
                // else it is stored, and this pair finishes the tile only if it turns out to be the last after all.
                // Flags go through one of four sets taken in turn: a set is not rewritten while a slower warp reads it.
                unsigned *counter = a.counters + 2 * u + int(rank);
                const unsigned others = unsigned(c_last - c_first);
                volatile uint32_t *fl = fold_flags + (flag_turn & 3);
                if (tid == 0) {
                    const unsigned seen = *reinterpret_cast<volatile unsigned *>(counter);
                    __threadfence();
                    *fl = seen == others ? 1u : 0u;
                }
                if (!(ok = epi_sync())) break;
                mine = *fl != 0u;
                ++flag_turn;
                if (!mine) {
                    store_partial<NT>(o, acc, col_grp, kEpiWarps / 4);
                    // The barrier orders every thread's stores before thread 0's fence, which is cumulative.
                    if (!(ok = epi_sync())) break;
                    fl = fold_flags + (flag_turn & 3);
                    if (tid == 0) {
                        __threadfence();
                        *fl = atomicAdd(counter, 1u) == others ? 1u : 0u;
                    }
                    if (!(ok = epi_sync())) break;
                    mine = *fl != 0u;
                    ++flag_turn;
                }
                if (mine) {
                    __threadfence();
                    if (tid == 0) *counter = 0u;
                }
            }
            // The conversion warps are done when the range's last tile is, and take their share of its columns.
            if (last && tid == 0) {
                last_flags[0] = mine ? 1u : 0u;
                last_flags[1] = uint32_t(c_first);
                last_flags[2] = uint32_t(c_last);
                mbar_arrive(last_fold);
            }
            if (mine)
                finish_tile<NT>(a, o, acc, col_grp, (last ? kEpiWarps + kConvWarps : kEpiWarps) / 4, c_first, c_last, pair, rank,
                            lane_grp * 32 + lane);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) arrive_cluster(acc_empty_lead);
            f = seg_end;
        }
    }
    if (!ok) {
        *abort_flag = 1u;
        atomicExch(a.status, kDevTimeout);
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (tid == 0 && *abort_flag != 0u)
        for (uint32_t r = 0; r < 2; ++r) store_in_cta(smem_u32(const_cast<uint32_t *>(pair_abort + rank)), r, 1u);
    __syncwarp();
    cluster_sync_all();  // neither CTA leaves while the other may still reach into it
    if ((pair_abort[0] | pair_abort[1]) != 0u) {
        if (rank == 0 && tid == 0) drain_activations(b_full, AS, F::b_stage, int(pair_issued[0]), int(pair_issued[1]));
        __syncwarp();
        cluster_sync_all();
    }
    if (warp == kEpiWarps + kConvWarps)
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_d), "r"(kWideTmemCols) : "memory");
}

template <int TYPE, int NT>
cudaError_t launch_form(const GemmArgs &a, cudaStream_t stream) {
    long long tiles = 0;
    for (int s = 0; s < a.nseg; ++s) tiles += (a.seg[s].rows + kPairM - 1) / kPairM;
    const long long units = tiles * ((a.n + NT - 1) / NT), raw_total = a.cols / kRawK, total = units * raw_total;
    const long long most = (a.sm_count > 1 ? a.sm_count : 148) / 2;
    long long pairs = total / 2 < most ? (total / 2 > 0 ? total / 2 : 1) : most;
    // Fewer tiles than pairs: a whole number of pairs per tile, so that a pair takes part in one partial tile instead of
    // two, unless that leaves more than a fifth of the pairs idle (4096 x 4096 against 512 rows, 64 of 74 pairs: 41.0 us,
    // 44.9 us cut into 74 ranges; 6144 rows would leave 26 idle).
    if (units < pairs) {
        long long per = pairs / units;
        if (per > raw_total / 2) per = raw_total / 2 > 0 ? raw_total / 2 : 1;
        if (units * per * 5 >= pairs * 4) pairs = units * per;
    }
    if (total * pairs >= (1ll << 32)) return cudaErrorInvalidValue;  // the kernel's work-list arithmetic is 32-bit
    if (a.scratch == nullptr || a.counters == nullptr || 2 * units > a.counters_len ||
        size_t(pairs) * 4 * kTileM * kMaxN > a.scratch_floats)
        return cudaErrorInvalidValue;
    CUtensorMap maps[4];
    for (int s = 0; s < 3; ++s) memcpy(&maps[s], a.seg[s < a.nseg ? s : 0].tmap->bytes, sizeof(CUtensorMap));
    memcpy(&maps[3], a.xmap->bytes, sizeof(CUtensorMap));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(2 * pairs));
    cfg.blockDim = dim3(kWideThreads);
    cfg.dynamicSmemBytes = WideSmem<TYPE, NT>::total;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = a.programmatic ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, gemm_wide_kernel<TYPE, NT>, a, maps[0], maps[1], maps[2], maps[3]);
}

template <int TYPE>
cudaError_t launch_wide(const GemmArgs &a, cudaStream_t stream) {
    return gemm_wide_tile(a.n) == 192 ? launch_form<TYPE, 192>(a, stream) : launch_form<TYPE, 256>(a, stream);
}

template <int TYPE>
cudaError_t configure_wide() {
    const cudaError_t e = cudaFuncSetAttribute(gemm_wide_kernel<TYPE, 192>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               WideSmem<TYPE, 192>::total);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(gemm_wide_kernel<TYPE, 256>, cudaFuncAttributeMaxDynamicSharedMemorySize, WideSmem<TYPE, 256>::total);
}

}  // namespace

// Both sides are measured at the head of this file.
int gemm_wide_tile(int n) { return n > 192 && n <= 256 ? 256 : 192; }

cudaError_t gemm_wide_configure() {
    cudaError_t e;
    if ((e = configure_wide<kQ4_K>()) != cudaSuccess) return e;
    if ((e = configure_wide<kQ4_0>()) != cudaSuccess) return e;
    if ((e = configure_wide<kQ6_K>()) != cudaSuccess) return e;
    if ((e = configure_wide<kQ5_K>()) != cudaSuccess) return e;
    if ((e = configure_wide<kQ4_1>()) != cudaSuccess) return e;
    return configure_wide<kQ8_0>();
}

cudaError_t gemm_wide_launch(const GemmArgs &a, cudaStream_t stream) {
    switch (a.type) {
        case kQ4_K: return launch_wide<kQ4_K>(a, stream);
        case kQ4_0: return launch_wide<kQ4_0>(a, stream);
        case kQ8_0: return launch_wide<kQ8_0>(a, stream);
        case kQ6_K: return launch_wide<kQ6_K>(a, stream);
        case kQ5_K: return launch_wide<kQ5_K>(a, stream);
        case kQ4_1: return launch_wide<kQ4_1>(a, stream);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace jl
