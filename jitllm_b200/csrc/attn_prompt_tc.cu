// Prompt attention on the 5th-generation tensor cores: the rows of one prompt chunk (one sequence, keys already in the
// pages) against all keys up to each row's own. The rotated query in two binary16 parts (hi + lo, 22 bits) against binary16
// keys, binary32 scores, running maximum and sum, probabilities rounded to binary16 against binary16 values, binary32 sums
// (inference/op/CpuOperations.java:94-235 is what it computes; function of the reference's tensor-core prompt attention,
// backend/tornado/layers/TensorCoreBatchAttention.java:227-366, not its code).
//
// A CTA takes 128 / G query rows and the G query heads of one KV head: 128 rows that share every key. Per tile of 128
// keys: S = Qlo K^T + Qhi K^T (both operands in shared memory, 128-byte swizzle, S in tensor memory, two buffers),
// softmax by 256 threads (a row per lane, two threads per row), P as binary16 back into tensor memory, O = P V with V as
// it lies in the pages (the B operand is "MN-major", so nothing is transposed), and the tile's O is added to registers
// scaled by the running maximum. The scores of tile t + 1 and the values of tile t - 1 are multiplied while the softmax
// of tile t runs.
//
// Measured (B200, one launch of 512 rows at the 8B shapes, cold L2) against the kernel before it, which multiplied with
// mma.sync from registers, read its rows' positions one after the other and stored two bytes at a time: 73 -> 42 us against
// the first 512 keys, 204 -> 92 us against 2048, 725 -> 293 us against 8192. Faster over the whole range, so there is one
// kernel. Distance from a 64-bit softmax (2-norm; standard deviation of the scores 1 to 12, common offset 0 to 2000, 512 to
// 8192 keys): 3.4e-5 to 2.0e-4, what the rounding of the probabilities leaves, and no more than that kernel's.
// What bounds it: 4.3 us per 128 keys against 0.8 us of tensor work and about 1.1 us of exponentials. Without copies after
// the second tile the 8192-token prompt was 7 % faster, without the exponentials 16 %: the softmax warps' chain (two passes
// over the scores, two row barriers, adding the tile's O) comes first, then the copies.
// The tensor-memory instructions and the row barriers are .sync.aligned: each follows a __syncwarp() or a vote behind whatever
// may have split the warp (a lane's arrival, a poll that lanes leave at different times).
// Roles: warps 0-7 softmax and output, warps 8-9 copy keys, 10-11 values (cp.async, a ring of two tiles each), warp 12
// issues the MMAs. They meet at mbarriers; every wait is bounded and a wait that runs out sets the status word.
#include "gemm_tc_core.cuh"
#include "ops.cuh"

namespace jl {
namespace {

constexpr int kPtRows = 128, kPtKeys = 128;
constexpr int kPtSoftWarps = 8, kPtThreads = 13 * 32;
constexpr uint32_t kPtS = 0, kPtO = 256, kPtP = 384, kPtCols = 512;  // tensor-memory columns: two S buffers, O, P
constexpr int kPtPages = 1024;  // page bases kept in shared memory (16 K keys of 16-token pages)

template <int HD>
struct PtSmem {
    static constexpr int atom = kPtKeys * 128;           // 64 dimensions of 128 rows or keys
    static constexpr int tile = atom * (HD / 64);
    static constexpr int q_off = 0;                       // hi, then lo
    static constexpr int k_off = 2 * tile, v_off = k_off + 2 * tile;
    static constexpr int pages_off = v_off + 2 * tile;
    static constexpr int xch_off = pages_off + kPtPages * 8;
    static constexpr int bar_off = xch_off + 2 * kPtRows * 4;
    static constexpr int total = bar_off + 256 + 1024;
    static_assert(total <= 227 * 1024, "shared memory budget");
};

__device__ __forceinline__ void pt_cp_async(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ float pt_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// One MMA (or commit) by an elected lane of a converged warp: its operands are warp-uniform.
__device__ __forceinline__ void umma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, pe;\n\telect.sync _|pe, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "@pe tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void umma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, pe;\n\telect.sync _|pe, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "@pe tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void umma_commit_one(uint64_t *bar) {
    asm volatile(
        "{\n\t.reg .pred pe;\n\telect.sync _|pe, 0xffffffff;\n\t"
        "@pe tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_u32(bar)) : "memory");
}
// 128-byte swizzle, groups of eight rows 1024 B apart; lead: the stride between 64-element blocks along the contiguous
// dimension (MN-major operands; unused by K-major ones), in bytes.
__device__ __forceinline__ uint64_t pt_desc(uint32_t addr, uint32_t lead) {
    const uint32_t lo = ((addr >> 4) & 0x3FFFu) | ((lead >> 4) << 16);
    const uint32_t hi = uint32_t(1024 >> 4) | (1u << 14) | (2u << 29);
    return (uint64_t(hi) << 32) | lo;
}

template <int HD, int G>
__global__ void __launch_bounds__(kPtThreads, 1) attn_prompt_tc_kernel(const AttnArgs a, int n) {
    using S = PtSmem<HD>;
    constexpr int RQ = kPtRows / G;  // query rows per CTA
    extern __shared__ uint8_t smem_raw[];
    uint8_t *base = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    int64_t *page_base = reinterpret_cast<int64_t *>(base + S::pages_off);
    float *xch = reinterpret_cast<float *>(base + S::xch_off);  // [2][128]
    uint64_t *bars = reinterpret_cast<uint64_t *>(base + S::bar_off);
    uint64_t *k_full = bars, *k_empty = bars + 2, *v_full = bars + 4, *v_empty = bars + 6;  // [2] each
    uint64_t *s_full = bars + 8, *s_empty = bars + 10;                                     // [2] each
    uint64_t *p_full = bars + 12, *o_full = bars + 13, *q_full = bars + 14;
    uint32_t *tmem_ptr = reinterpret_cast<uint32_t *>(bars + 16);
    volatile uint32_t *abort_flag = tmem_ptr + 1;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int kvh = blockIdx.y, cta_row0 = blockIdx.x * RQ;

    if (warp == 12) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_ptr)), "r"(kPtCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(k_full + i, 2);
            mbar_init(k_empty + i, 1);
            mbar_init(v_full + i, 2);
            mbar_init(v_empty + i, 1);
            mbar_init(s_full + i, 1);
            mbar_init(s_empty + i, kPtSoftWarps);
        }
        mbar_init(p_full, kPtSoftWarps);
        mbar_init(o_full, 1);
        mbar_init(q_full, kPtSoftWarps);
        mbar_fence_init();
        *abort_flag = 0u;
    }
    // Positions, slots, the activity flags and the block table are not written by anything in this step: what follows
    // from them is worked out while the kernel ahead still runs. Keys this CTA needs: up to its rows' largest position.
    const int slot = a.slots[cta_row0];
    int last = -1;
    for (int r = cta_row0 + lane; r < min(n, cta_row0 + RQ); r += 32)
        if (a.active == nullptr || a.active[r] != 0) last = max(last, a.positions[r]);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) last = max(last, __shfl_xor_sync(0xffffffffu, last, off));
    const int tiles = last / kPtKeys + (last >= 0 ? 1 : 0);
    const int bt = a.kv.block_tokens;
    const int64_t block_stride = int64_t(a.kv.layers) * bt * a.kv.kv_dim;
    const auto page_start = [&](int pg) {
        const int64_t phys = a.kv.block_table[int64_t(slot) * a.kv.blocks_per_slot + pg];
        return phys * block_stride + int64_t(a.layer) * bt * a.kv.kv_dim + int64_t(kvh) * HD;
    };
    const int npages = last >= 0 ? last / bt + 1 : 0;
    for (int pg = tid; pg < min(npages, kPtPages); pg += kPtThreads) page_base[pg] = page_start(pg);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_ptr;
    // Only now: a dependent kernel's CTA that came to this SM ahead of the allocation could take the tensor memory and then
    // wait for this grid, which would wait for it.
    pdl_launch_dependents();
    bool ok = true;

    if (warp == 12) {
        // ---- MMA issue -----------------------------------------------------------------------------------
        if (tiles > 0) {
            constexpr uint32_t idesc_s = (1u << 4) | (uint32_t(kPtKeys >> 3) << 17) | (uint32_t(kPtRows >> 4) << 24);
            constexpr uint32_t idesc_o = (1u << 4) | (1u << 16) | (uint32_t(HD >> 3) << 17) | (uint32_t(kPtRows >> 4) << 24);
            const uint32_t q0 = smem_u32(base + S::q_off), k0 = smem_u32(base + S::k_off), v0 = smem_u32(base + S::v_off);
            int keys_in = 0, values_in = 0;  // tiles whose MMAs have been issued
            ok = __all_sync(0xffffffffu, mbar_poll_bounded(q_full, 0));
            for (int t = 0; t <= tiles && ok && *abort_flag == 0u; ++t) {
                const int b = t & 1;
                if (t < tiles) {
                    ok = mbar_spin_bounded(k_full + b, uint32_t(t >> 1) & 1u);
                    if (ok && t >= 2) ok = mbar_spin_bounded(s_empty + b, uint32_t((t >> 1) - 1) & 1u);
                    if (!__all_sync(0xffffffffu, ok)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    // The lo part first: every addition is cut off at the accumulator's last place, and the lo products
                    // (2^-11 of the hi ones) lose nothing that counts while the hi sum is not there yet.
#pragma unroll
                    for (int part = 0; part < 2; ++part) {
#pragma unroll
                        for (int k = 0; k < HD / 16; ++k) {
                            const uint32_t off = uint32_t(k >> 2) * S::atom + uint32_t(k & 3) * 32u;
                            umma_ss(tmem + kPtS + uint32_t(b) * kPtKeys, pt_desc(q0 + uint32_t(1 - part) * S::tile + off, 16),
                                    pt_desc(k0 + uint32_t(b) * S::tile + off, 16), idesc_s, part + k > 0 ? 1u : 0u);
                        }
                    }
                    umma_commit_one(s_full + b);
                    umma_commit_one(k_empty + b);
                    ++keys_in;
                }
                if (t > 0) {
                    const int pb = (t - 1) & 1;
                    ok = mbar_spin_bounded(v_full + pb, uint32_t((t - 1) >> 1) & 1u) &&
                         mbar_spin_bounded(p_full, uint32_t(t - 1) & 1u);  // P written, the O before it read out
                    if (!__all_sync(0xffffffffu, ok)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
#pragma unroll
                    for (int k = 0; k < kPtKeys / 16; ++k)
                        umma_ts(tmem + kPtO, tmem + kPtP + uint32_t(k) * 8u,
                                pt_desc(v0 + uint32_t(pb) * S::tile + uint32_t(k) * 2048u, S::atom), idesc_o, k > 0 ? 1u : 0u);
                    umma_commit_one(o_full);
                    umma_commit_one(v_empty + pb);
                    ++values_in;
                }
            }
            // The MMAs are over and the last hand-backs have arrived before this CTA leaves, whatever ended the loop.
            for (int t = max(keys_in - 2, 0); t < keys_in; ++t) ok = mbar_poll_bounded(k_empty + (t & 1), uint32_t(t >> 1) & 1u) && ok;
            for (int t = max(values_in - 2, 0); t < values_in; ++t) ok = mbar_poll_bounded(v_empty + (t & 1), uint32_t(t >> 1) & 1u) && ok;
        }
    } else if (warp >= kPtSoftWarps) {
        // ---- key and value tiles, past the last key zeros -------------------------------------------------
        pdl_wait();
        const bool vals = warp >= kPtSoftWarps + 2;
        const int lt = tid - (kPtSoftWarps + (vals ? 2 : 0)) * 32;  // 0..63
        const __half *pool = vals ? a.kv.vpool : a.kv.kpool;
        uint64_t *full = vals ? v_full : k_full, *empty = vals ? v_empty : k_empty;
        const uint32_t ring = smem_u32(base + (vals ? S::v_off : S::k_off));
        constexpr int kParts = HD / 8, kPerPass = 64 / kParts;
        const int part = lt % kParts, key0 = lt / kParts;
        const uint32_t dst0 = ring + uint32_t(part >> 3) * S::atom;
        // This thread copies the same 16-byte part of every kPerPass-th key; its page and place in the page move on by
        // additions (a division per copy made these warps the slowest part of the kernel).
        int at = key0, pg = key0 / bt, within = key0 - pg * bt;
        const __half *page = nullptr;
        const auto find_page = [&]() {
            if (at <= last) page = pool + (pg < kPtPages ? page_base[pg] : page_start(pg)) + part * 8;
        };
        find_page();
        for (int t = 0; t < tiles && *abort_flag == 0u; ++t) {
            if (t >= 2) ok = mbar_poll_bounded(empty + (t & 1), uint32_t((t >> 1) - 1) & 1u);
            if (!__all_sync(0xffffffffu, ok)) {
                ok = false;
                break;
            }
            const uint32_t dst = dst0 + uint32_t(t & 1) * S::tile;
#pragma unroll 8
            for (int i = 0; i < kPtKeys / kPerPass; ++i) {
                const int key = key0 + i * kPerPass;
                const uint32_t to = dst + uint32_t(key) * 128u + uint32_t(((part & 7) ^ (key & 7)) << 4);
                if (at <= last)
                    pt_cp_async(to, page + int64_t(within) * a.kv.kv_dim);
                else
                    asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(to), "r"(0u) : "memory");
                at += kPerPass;
                within += kPerPass;
                if (within >= bt) {
                    do {
                        within -= bt;
                        ++pg;
                    } while (within >= bt);
                    find_page();
                }
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(full + (t & 1));
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else {
        // ---- softmax and output: row (warp & 3) * 32 + lane, half (warp >> 2) of the keys and dimensions ----
        pdl_wait();
        const int r = (warp & 3) * 32 + lane, half = warp >> 2;
        const int row = cta_row0 + r / G, head = kvh * G + r % G;
        const bool on = row < n && (a.active == nullptr || a.active[row] != 0);
        const int pos = on ? a.positions[row] : -1;
        constexpr int kDims = HD / 2;  // dimensions of this thread
        {
            const float *q = a.q + size_t(row) * a.dim + size_t(head) * HD;
#pragma unroll
            for (int c = 0; c < kDims / 8; ++c) {
                const int d = half * kDims + c * 8;
                float x[8];
                if (on) {
                    const float4 v0 = *reinterpret_cast<const float4 *>(q + d), v1 = *reinterpret_cast<const float4 *>(q + d + 4);
                    const float4 cr = *reinterpret_cast<const float4 *>(a.rope_cos + size_t(pos) * (HD / 2) + d / 2);
                    const float4 ci = *reinterpret_cast<const float4 *>(a.rope_sin + size_t(pos) * (HD / 2) + d / 2);
                    const float in[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
                    const float co[4] = {cr.x, cr.y, cr.z, cr.w}, si[4] = {ci.x, ci.y, ci.z, ci.w};
#pragma unroll
                    for (int p = 0; p < 4; ++p) {
                        x[2 * p] = __fsub_rn(__fmul_rn(in[2 * p], co[p]), __fmul_rn(in[2 * p + 1], si[p]));
                        x[2 * p + 1] = __fadd_rn(__fmul_rn(in[2 * p], si[p]), __fmul_rn(in[2 * p + 1], co[p]));
                    }
                } else {
#pragma unroll
                    for (int p = 0; p < 8; ++p) x[p] = 0.f;
                }
                uint32_t hi[4], lo[4];
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    const __half2 h = __floats2half2_rn(x[2 * p], x[2 * p + 1]);
                    const float2 back = __half22float2(h);
                    const __half2 l = __floats2half2_rn(x[2 * p] - back.x, x[2 * p + 1] - back.y);
                    hi[p] = h2_bits(h);
                    lo[p] = h2_bits(l);
                }
                const uint32_t to = uint32_t(d >> 6) * S::atom + sw128_offset(r, (d & 63) >> 3);
                *reinterpret_cast<uint4 *>(base + S::q_off + to) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                *reinterpret_cast<uint4 *>(base + S::q_off + S::tile + to) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(q_full);
        }
        float o[kDims];
#pragma unroll
        for (int d = 0; d < kDims; ++d) o[d] = 0.f;
        float m = -INFINITY, l = 0.f, corr = 1.0f;  // corr: what the sums before the tile in flight are scaled by
        // exp(s / sqrt(HD) - max) = 2^(s * scale - sub), sub = max * scale rounded: one fused multiply-add and one ex2 per score.
        // Its relative error is 2^-22 of the ex2 and up to |sub| 2^-25 of the rounding of sub. The latter is common to all
        // keys and leaves with the division, because the sums of earlier tiles are moved from one rounded sub to the next.
        float sub = 0.f;
        const float scale = 1.4426950408889634f / sqrtf(static_cast<float>(HD));
        const uint32_t lanes = uint32_t((warp & 3) * 32) << 16;
        // the two warps that share these 32 rows
        const auto row_sync = [&]() {
            __syncwarp();
            asm volatile("bar.sync %0, 64;" ::"r"(1 + (warp & 3)) : "memory");
        };
        // A wait that ran out is noted, and the loop goes on to its end so that the two warps of a row stay in step; later
        // waits poll once, and nothing it computes is used (the status word is set).
        bool all_ok = true;
        const auto add_o = [&](int t) {  // o = o * corr + the O of tile t
            ok = mbar_spin_bounded(o_full, uint32_t(t) & 1u, all_ok ? (1u << 26) : 1u);
            __syncwarp();
            tc_fence_after();
#pragma unroll
            for (int g = 0; g < kDims / 16; ++g) {
                float v[16];
                tmem_ld16(tmem + lanes + kPtO + uint32_t(half * kDims + g * 16), v);
#pragma unroll
                for (int j = 0; j < 16; ++j) o[g * 16 + j] = o[g * 16 + j] * corr + v[j];
            }
        };
        for (int t = 0; t < tiles; ++t) {
            ok = mbar_spin_bounded(s_full + (t & 1), uint32_t(t >> 1) & 1u, all_ok ? (1u << 26) : 1u);
            all_ok = all_ok && ok;
            __syncwarp();
            tc_fence_after();
            // The scores are read twice, for the maximum and for the exponentials: with the 64 sums they do not fit the
            // registers at once (128 a thread: one scheduler holds four of the thirteen warps).
            const uint32_t s_cols = tmem + lanes + kPtS + uint32_t((t & 1) * kPtKeys + half * 64);
            const int key0 = t * kPtKeys + half * 64;
            const bool masked = __any_sync(0xffffffffu, key0 + 63 > pos);  // the warp decides: the usual tile needs no masks
            const int limit = pos - key0;
            float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                float v[16];
                tmem_ld16(s_cols + uint32_t(g * 16), v);
                if (masked) {
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (g * 16 + j > limit) v[j] = -INFINITY;
                }
#pragma unroll
                for (int j = 0; j < 16; ++j) mx4[j & 3] = fmaxf(mx4[j & 3], v[j]);
            }
            const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
            xch[half * kPtRows + r] = mx;
            row_sync();
            const float mn = fmaxf(m, fmaxf(mx, xch[(half ^ 1) * kPtRows + r]));
            const float next_sub = mn == -INFINITY ? 0.f : mn * scale;  // -inf: nothing but masked keys so far
            const float next_corr = m == -INFINITY ? 0.f : pt_exp2(sub - next_sub);  // before the first key the sums are 0
            m = mn;
            sub = next_sub;
            l *= next_corr;
            uint32_t p[32];
            float sum4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                float v[16];
                tmem_ld16(s_cols + uint32_t(g * 16), v);
                if (masked) {
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (g * 16 + j > limit) v[j] = -INFINITY;
                }
#pragma unroll
                for (int j = 0; j < 16; j += 2) {
                    const float p0 = pt_exp2(fmaf(v[j], scale, -sub)), p1 = pt_exp2(fmaf(v[j + 1], scale, -sub));
                    const __half2 ph = __floats2half2_rn(p0, p1);
                    const float2 pr = __half22float2(ph);  // the sum is over what the values are multiplied by
                    sum4[j & 2] += pr.x;
                    sum4[(j & 2) + 1] += pr.y;
                    p[(g * 16 + j) / 2] = h2_bits(ph);
                }
            }
            l += (sum4[0] + sum4[1]) + (sum4[2] + sum4[3]);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(s_empty + (t & 1));
            if (t > 0) add_o(t - 1);
            all_ok = all_ok && ok;
            corr = next_corr;
            __syncwarp();
            {
                uint32_t c[16];
#pragma unroll
                for (int g = 0; g < 2; ++g) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) c[j] = p[g * 16 + j];
                    tmem_st16(tmem + lanes + kPtP + uint32_t(half * 32 + g * 16), c);
                }
            }
            tmem_wait_st();
            tc_fence_before();
            row_sync();  // both halves have read the maxima: xch may be rewritten
            if (lane == 0) mbar_arrive(p_full);
        }
        if (tiles > 0) {
            add_o(tiles - 1);
            all_ok = all_ok && ok;
        }
        ok = all_ok;
        xch[half * kPtRows + r] = l;
        row_sync();
        l += xch[(half ^ 1) * kPtRows + r];
        if (on) {
            const size_t at = size_t(row) * a.dim + size_t(head) * HD + half * kDims;
#pragma unroll
            for (int d = 0; d < kDims; d += 4) {
                const float4 v = make_float4(o[d] / l, o[d + 1] / l, o[d + 2] / l, o[d + 3] / l);
                *reinterpret_cast<float4 *>(a.out + at + d) = v;
                if (a.out_hi != nullptr) {  // operand order: pairs (k0, k2), (k1, k3) inside every four
                    const __half2 h0 = __floats2half2_rn(v.x, v.z), h1 = __floats2half2_rn(v.y, v.w);
                    const float2 b0 = __half22float2(h0), b1 = __half22float2(h1);
                    const __half2 l0 = __floats2half2_rn(v.x - b0.x, v.z - b0.y), l1 = __floats2half2_rn(v.y - b1.x, v.w - b1.y);
                    *reinterpret_cast<uint2 *>(static_cast<__half *>(a.out_hi) + at + d) = make_uint2(h2_bits(h0), h2_bits(h1));
                    *reinterpret_cast<uint2 *>(static_cast<__half *>(a.out_lo) + at + d) = make_uint2(h2_bits(l0), h2_bits(l1));
                }
            }
        }
    }
    if (!ok) {
        *abort_flag = 1u;
        if (a.status != nullptr) atomicExch(a.status, kDevTimeout);
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 12) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kPtCols) : "memory");
}

template <int HD, int G>
cudaError_t launch_t(const AttnArgs &a, int n, cudaStream_t stream, bool programmatic) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned((n + kPtRows / G - 1) / (kPtRows / G)), unsigned(a.kv_heads));
    cfg.blockDim = dim3(kPtThreads);
    cfg.dynamicSmemBytes = PtSmem<HD>::total;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = programmatic ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, attn_prompt_tc_kernel<HD, G>, a, n);
}
template <int HD>
cudaError_t launch_hd(const AttnArgs &a, int n, cudaStream_t s, bool pdl) {
    switch (a.heads / a.kv_heads) {
        case 1: return launch_t<HD, 1>(a, n, s, pdl);
        case 2: return launch_t<HD, 2>(a, n, s, pdl);
        case 4: return launch_t<HD, 4>(a, n, s, pdl);
        case 8: return launch_t<HD, 8>(a, n, s, pdl);
        default: return cudaErrorInvalidValue;
    }
}
template <int HD, int G>
cudaError_t configure_t() {
    return cudaFuncSetAttribute(attn_prompt_tc_kernel<HD, G>, cudaFuncAttributeMaxDynamicSharedMemorySize, PtSmem<HD>::total);
}
template <int HD>
cudaError_t configure_hd() {
    cudaError_t e;
    if ((e = configure_t<HD, 1>()) != cudaSuccess) return e;
    if ((e = configure_t<HD, 2>()) != cudaSuccess) return e;
    if ((e = configure_t<HD, 4>()) != cudaSuccess) return e;
    return configure_t<HD, 8>();
}

}  // namespace

cudaError_t attention_prompt_configure() {
    const cudaError_t e = configure_hd<128>();
    return e != cudaSuccess ? e : configure_hd<64>();
}

cudaError_t attention_prompt_launch(const AttnArgs &a, int n, cudaStream_t stream, bool programmatic) {
    if (a.head_dim == 128) return launch_hd<128>(a, n, stream, programmatic);
    if (a.head_dim == 64) return launch_hd<64>(a, n, stream, programmatic);
    return cudaErrorInvalidValue;
}

}  // namespace jl
