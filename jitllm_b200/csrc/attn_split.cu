// RoPE + KV append + paged decode attention with the keys of a sequence split over CTAs (sm_100a), for launches that have
// fewer (row, KV head) pairs than the GPU has room for.
//
// What it computes: CpuOperations.rope + appendKeyValue + attention (inference/op/CpuOperations.java:94-204), softmax online;
// K and V are rounded to binary16 on append exactly as ArrayHalfFloatTensor.setFloat does
// (tensor/standard/ArrayHalfFloatTensor.java:33-40).
//
// One CTA of eight warps = (range of keys, KV head, row). The G query heads that share the KV head are rows of one MMA
// tile: a query, scaled by a power of two from its head's largest element, and a probability are each the sum of three
// binary16 parts, which are three rows each (3 G <= 12 of the 16 rows; G = 8 takes two tiles), so q.k and p.v keep their 32
// bits (split3 says down to which size) while keys and values are binary16 as stored. Tiles of 64 keys come through a double
// buffer by cp.async; warp w multiplies sixteen of a tile's keys and half of the output dimensions. A launch is latency: 64
// keys per CTA as long as there are CTAs, then longer ranges. The last CTA of a (row, KV head) to finish folds the ranges'
// results; the arrival is one atomic.
// Error against a 64-bit softmax over the same query, keys and values (2-norm; geometric mean over 20 models, head sizes 64
// and 128, groups of 2, 4 and 8, scores of standard deviation 0.2 to 8, 1 to 3000 keys): 1.46e-7; scalar binary32 sums in the
// split of the keys that a kernel of scalar products would take 1.50e-7. It does not depend on the size of the queries
// (2^-4 to 2^-12 times the usual one, keys as much larger: 2.4e-7 where it is 2.5e-7), nor on how the heads of a group compare.
#include "ops.cuh"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

namespace jl {

JL_TRACE_DEFINE_BIND(attn_split_trace_bind)

namespace {

constexpr int kThreads = 256;
constexpr int kTile = 64;         // keys
constexpr int kGroups = kTile / 16;
constexpr int kKeysPerSplit = 64;
constexpr int kPages = 512;       // page numbers kept in shared memory

__device__ __forceinline__ void mma_f16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldmatrix4_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory"); }
// x, at most 2^15 in magnitude, as the sum of three binary16 values of eight significant bits each: all 24 bits from 1/2 up, and
// below that all of them down to 2^-24, where binary16 ends (what is lost is at most 2^-25). The callers scale what they split by
// a power of two so that its largest lies between 2^14 and 2^15: every value down to 2^-15 of the largest is whole, and what the
// smaller ones lose is at most 2^-39 of the largest. (Parts of eight bits, not of eleven: the tensor core cuts its sums of sixteen
// products off at some 2^-24 of the largest, and a part's products with binary16 keys would reach below that. Eight bits leave
// the first part's sums whole, and what is cut off the other two is 2^-8 and 2^-16 of it.)
__device__ __forceinline__ void split3(float x, __half (&h)[3]) {
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        h[p] = __float2half_rn(__bfloat162float(__float2bfloat16_rn(x)));
        x -= __half2float(h[p]);  // exact; with what binary16 dropped of the part
    }
    h[2] = __float2half_rn(x);
}
// The power of two that takes a largest magnitude (its bits, finite) to between 2^14 and 2^15, as bits; 2^100 for those below 2^-86,
// whose scores are all but equal.
__device__ __forceinline__ unsigned query_scale(unsigned most) { return min(268u - (most >> 23), 227u) << 23; }
// The sum of 2^n values in n roundings.
template <int N>
__device__ __forceinline__ float sum_pairs(const float (&x)[N]) {
    float s[N];
#pragma unroll
    for (int i = 0; i < N; ++i) s[i] = x[i];
#pragma unroll
    for (int w = 1; w < N; w *= 2)
#pragma unroll
        for (int i = 0; i < N; i += 2 * w) s[i] += s[i + w];
    return s[0];
}

template <int HD, int G>
struct SplitAttn {
    static constexpr int LD = HD + 8;          // halves per row: no bank conflicts
    static constexpr int QT = G == 8 ? 2 : 1;  // sixteen-row tiles that hold three parts of G heads
    // The row of a head's part. The sum over the parts starts with rows r and r + 8: the two small parts meet first, so that the
    // large one is rounded once.
    static __host__ __device__ constexpr int row(int part, int g) { return part < 2 ? part * G + g : G == 8 ? 16 + g : 8 + G + g; }
    struct Smem {
        alignas(16) __half q[QT * 16][LD];
        int pages[kPages];
        float w[kGroups][G];  // merge weights
        unsigned q_most[G * HD / 64];  // the largest finite magnitude of every 64 elements of the rotated queries, as bits
        float inv[G], sum[G], top[G];
        int is_last;
        union {
            struct {
                alignas(16) __half k[2][kTile][LD];
                alignas(16) __half v[2][kTile][LD];
            } tile;
            float merge[kGroups][G][HD + 2];
            float fold[1024];  // [range][head] maxima, then weights
        };
    };
};

// The keys of one CTA: start .. stop - 1 from the pages; the last range of a decode launch also has this step's own key, behind them.
struct KeyRange {
    int nsplit, start, stop;
    bool owns_new;
};
__device__ __forceinline__ KeyRange key_range(const AttnArgs &a, int split, int pos) {
    const int old = a.append != 0 ? pos : pos + 1;  // keys in the pages
    KeyRange r;
    r.nsplit = max(1, min(a.nsplit, (old + kKeysPerSplit - 1) / kKeysPerSplit));
    const int chunk = (old + r.nsplit - 1) / r.nsplit;
    r.start = min(old, split * chunk);
    r.stop = min(old, r.start + chunk);
    r.owns_new = a.append != 0 && split == r.nsplit - 1;
    return r;
}

// The CTA's range once more, in scalar binary32, when an infinity or NaN showed in its output: a zero part of a query or
// probability, or a row of the tile that holds no part, makes NaN of an infinite key or value, and so do parts of opposite signs.
// Here, as in the reference, a score of -inf has no weight, an infinite value gives an infinite output, and a NaN score reaches the
// output. Its speed matters to nobody: keys beyond 65504 do not occur in a model that works. Warp w takes every fourth key for
// half of the heads; the results go to the merge area as the tiles' do. Ends with that area written, no barrier. A call, and one
// that takes nothing from the caller's registers: in line it cost the launches that never get here 0.3 to 0.5 us in batches.
template <int HD, int G>
__device__ __noinline__ void scalar_range(const AttnArgs &a, typename SplitAttn<HD, G>::Smem &sm) {
    const int kvh = blockIdx.y, b = blockIdx.z, pos = a.positions[b], slot = a.slots[b];
    const KeyRange keys = key_range(a, blockIdx.x, pos);
    const int end = keys.stop + (keys.owns_new ? 1 : 0);
    constexpr int PAIRS = HD / 64;  // pairs of dimensions per lane
    const int lane = threadIdx.x & 31, kg = (threadIdx.x >> 5) % kGroups, half = (threadIdx.x >> 5) / kGroups;
    const int bt = a.kv.block_tokens, kv_dim = a.kv.kv_dim;
    const int32_t *table = a.kv.block_table + int64_t(slot) * a.kv.blocks_per_slot;
    const float inv_sqrt = 1.0f / sqrtf(static_cast<float>(HD));
    for (int g = half; g < G; g += 2) {
        float2 q[PAIRS], o[PAIRS];
#pragma unroll
        for (int i = 0; i < PAIRS; ++i) {
            const int p = lane + 32 * i;
            const float2 x = __ldcg(reinterpret_cast<const float2 *>(a.q + size_t(b) * a.dim + size_t(kvh * G + g) * HD) + p);
            const float c = a.rope_cos[size_t(pos) * (HD / 2) + p], s = a.rope_sin[size_t(pos) * (HD / 2) + p];
            q[i] = make_float2(__fsub_rn(__fmul_rn(x.x, c), __fmul_rn(x.y, s)), __fadd_rn(__fmul_rn(x.x, s), __fmul_rn(x.y, c)));
            o[i] = make_float2(0.f, 0.f);
        }
        float m = -INFINITY, l = 0.f;
        for (int t = keys.start + kg; t < end; t += kGroups) {
            const int64_t off = ((int64_t(table[t / bt]) * a.kv.layers + a.layer) * bt + t % bt) * kv_dim + int64_t(kvh) * HD;
            float2 v[PAIRS];
            float s = 0.f;
#pragma unroll
            for (int i = 0; i < PAIRS; ++i) {
                const float2 k = __half22float2(__ldcg(reinterpret_cast<const __half2 *>(a.kv.kpool + off) + lane + 32 * i));
                v[i] = __half22float2(__ldcg(reinterpret_cast<const __half2 *>(a.kv.vpool + off) + lane + 32 * i));
                s += q[i].x * k.x + q[i].y * k.y;
            }
            s = warp_sum(s) * inv_sqrt;
            const float mn = fmaxf(m, s), corr = mn == -INFINITY ? 1.0f : expf(m - mn), p = s == -INFINITY ? 0.f : expf(s - mn);
            m = mn;
            l = l * corr + p;
#pragma unroll
            for (int i = 0; i < PAIRS; ++i) {
                o[i].x = o[i].x * corr + p * v[i].x;
                o[i].y = o[i].y * corr + p * v[i].y;
            }
        }
#pragma unroll
        for (int i = 0; i < PAIRS; ++i) {
            sm.merge[kg][g][2 * (lane + 32 * i)] = o[i].x;
            sm.merge[kg][g][2 * (lane + 32 * i) + 1] = o[i].y;
        }
        if (lane == 0) {
            sm.merge[kg][g][HD] = m;
            sm.merge[kg][g][HD + 1] = l;
        }
    }
}

template <int HD, int G>
__global__ void __launch_bounds__(kThreads, 2) attn_split_kernel(const __grid_constant__ AttnArgs a) {
    using A = SplitAttn<HD, G>;
    constexpr int LD = A::LD, QT = A::QT, DB = HD / 16, ROW = HD + 2, PARTS = HD / 8;
    extern __shared__ __align__(16) uint8_t smem_raw[];
    typename A::Smem &sm = *reinterpret_cast<typename A::Smem *>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int split = blockIdx.x, kvh = blockIdx.y, b = blockIdx.z;
    const int trace = trace_begin(kTraceAttn);
    pdl_launch_dependents();
    const bool on = a.active == nullptr || a.active[b] != 0;
    const bool dec = a.append != 0;
    // A decode launch reads what no kernel of this step writes (position, slot, page table, old keys) before it waits for
    // the one that produces q, k and v: positions and slots are written by the host or by advance_kernel, and the kernel
    // after that one releases its dependents only when it has waited itself. The rows of a prompt wait first: their keys
    // were appended by the kernel ahead.
    if (!dec) pdl_wait();
    const int pos = on ? a.positions[b] : 0, slot = on ? a.slots[b] : 0;
    const KeyRange keys = key_range(a, split, pos);
    const int nsplit = keys.nsplit, start = keys.start, stop = keys.stop;
    if (!on || split >= nsplit) {
        if (dec) pdl_wait();
        return;
    }
    const bool owns_new = keys.owns_new;
    const int end = stop + (owns_new ? 1 : 0);
    const int bt = a.kv.block_tokens, kv_dim = a.kv.kv_dim;
    const int64_t block_stride = int64_t(a.kv.layers) * bt * kv_dim, in_layer = int64_t(a.layer) * bt * kv_dim + int64_t(kvh) * HD;
    const int32_t *table = a.kv.block_table + int64_t(slot) * a.kv.blocks_per_slot;
    const int first_page = start / bt, npages = stop > start ? (stop - 1) / bt - first_page + 1 : 0;
    for (int i = tid; i < min(npages, kPages); i += kThreads) sm.pages[i] = table[first_page + i];
    for (int i = tid; i < QT * 16 * LD / 2; i += kThreads) reinterpret_cast<uint32_t *>(&sm.q[0][0])[i] = 0u;
    constexpr int kPairs = (G + 2) * (HD / 2), kRounds = (kPairs + kThreads - 1) / kThreads;
    float cr[kRounds], ci[kRounds];  // of this thread's pairs of dimensions
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
        const int i = (tid + r * kThreads) % (HD / 2);
        cr[r] = a.rope_cos[size_t(pos) * (HD / 2) + i];
        ci[r] = a.rope_sin[size_t(pos) * (HD / 2) + i];
    }
    __syncthreads();
    const uint32_t k0 = smem_u32(&sm.tile.k[0][0][0]), v0 = smem_u32(&sm.tile.v[0][0][0]);
    auto load = [&](int t0, int buf) {
#pragma unroll
        for (int i = 0; i < kTile * PARTS / kThreads; ++i) {
            const int key = (i * kThreads + tid) / PARTS, part = tid % PARTS, t = t0 + key;
            const uint32_t at = uint32_t((buf * kTile + key) * LD + part * 8) * 2;
            if (t < stop) {
                const int pg = t / bt, in = pg - first_page;
                const int64_t off = int64_t(in < kPages ? sm.pages[in] : table[pg]) * block_stride + in_layer + int64_t(t - pg * bt) * kv_dim + part * 8;
                cp_async16(k0 + at, a.kv.kpool + off);
                cp_async16(v0 + at, a.kv.vpool + off);
            } else {
                sts64(k0 + at, 0u, 0u);
                sts64(k0 + at + 8, 0u, 0u);
                sts64(v0 + at, 0u, 0u);
                sts64(v0 + at + 8, 0u, 0u);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    load(start, 0);
    if (dec) pdl_wait();
    trace_mark(trace, 2);
    trace_word(trace, 6, trace_latest_exit());
    // Queries rotated, and the new key and value: rotated, rounded to binary16 as the append does.
    float qx[kRounds] = {}, qy[kRounds] = {};
    uint32_t fresh[kRounds] = {};
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
        const int idx = tid + r * kThreads, i = idx % (HD / 2);
        if (idx < G * (HD / 2)) {
            const float2 x = __ldcg(reinterpret_cast<const float2 *>(a.q + size_t(b) * a.dim + size_t(kvh * G + idx / (HD / 2)) * HD) + i);
            qx[r] = __fsub_rn(__fmul_rn(x.x, cr[r]), __fmul_rn(x.y, ci[r]));
            qy[r] = __fadd_rn(__fmul_rn(x.x, ci[r]), __fmul_rn(x.y, cr[r]));
            // the lanes of a warp have 64 elements of one head
            const unsigned ax = __float_as_uint(fabsf(qx[r])), ay = __float_as_uint(fabsf(qy[r])), inf = 0x7f800000u;
            const unsigned most = __reduce_max_sync(0xffffffffu, max(ax < inf ? ax : 0u, ay < inf ? ay : 0u));
            if (lane == 0) sm.q_most[idx / 32] = most;
        } else if (owns_new && idx < kPairs) {
            const bool is_k = idx < (G + 1) * (HD / 2);
            const float2 x = __ldcg(reinterpret_cast<const float2 *>((is_k ? a.k : a.v) + size_t(b) * kv_dim + size_t(kvh) * HD) + i);
            const __half2 h = is_k ? __halves2half2(__float2half_rn(__fsub_rn(__fmul_rn(x.x, cr[r]), __fmul_rn(x.y, ci[r]))),
                                                    __float2half_rn(__fadd_rn(__fmul_rn(x.x, ci[r]), __fmul_rn(x.y, cr[r]))))
                                   : __halves2half2(__float2half_rn(x.x), __float2half_rn(x.y));
            const int64_t off = int64_t(table[pos / bt]) * block_stride + in_layer + int64_t(pos % bt) * kv_dim;
            *reinterpret_cast<__half2 *>((is_k ? a.kv.kpool : a.kv.vpool) + off + 2 * i) = h;
            fresh[r] = *reinterpret_cast<const uint32_t *>(&h);
        }
    }
    // Every head's query is scaled by a power of two from its own largest element (the same for all ranges: they see the same
    // queries), so that the split keeps its bits whatever its magnitude and whatever its neighbours'.
    __syncthreads();
    auto scale_of = [&](int g) { return query_scale(HD == 64 ? sm.q_most[g] : max(sm.q_most[2 * g], sm.q_most[2 * g + 1])); };
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
        const int idx = tid + r * kThreads, i = idx % (HD / 2);
        if (idx < G * (HD / 2)) {
            const int g = idx / (HD / 2);
            __half p0[3], p1[3];
            const float scale = __uint_as_float(scale_of(g));
            split3(qx[r] * scale, p0);
            split3(qy[r] * scale, p1);
#pragma unroll
            for (int p = 0; p < 3; ++p) *reinterpret_cast<__half2 *>(&sm.q[A::row(p, g)][2 * i]) = __halves2half2(p0[p], p1[p]);
        }
    }
    trace_mark(trace, 3);
    const int gl = lane >> 2, t = lane & 3, kg = warp & (kGroups - 1), half = warp / kGroups;
    // 1 / sqrt(head size), and the scale of this lane's head taken back (exactly)
    const float to_score = (1.0f / sqrtf(static_cast<float>(HD))) * __uint_as_float((254u << 23) - scale_of(gl % G));
    constexpr float kUp = 32768.0f;  // probabilities, at most 1, are split as multiples of 2^-15
    float m = -INFINITY, l = 0.f, o[DB][4];
#pragma unroll
    for (int d = 0; d < DB; ++d) o[d][0] = o[d][1] = o[d][2] = o[d][3] = 0.f;
    // sum over the parts of a head: the lanes whose rows have the same head
    auto join = [&](float x) {
#pragma unroll
        for (int s = 4 * G; s < 32; s *= 2) x += __shfl_xor_sync(0xffffffffu, x, s);
        return x;
    };
    for (int t0 = start, buf = 0; t0 < end; t0 += kTile, buf ^= 1) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();  // the tile is there, and everybody is done with the other buffer
        if (t0 + kTile < end) load(t0 + kTile, buf ^ 1);
        if (owns_new && end - 1 - t0 < kTile) {  // the new key's tile
#pragma unroll
            for (int r = 0; r < kRounds; ++r) {
                const int idx = tid + r * kThreads, i = idx % (HD / 2);
                if (idx >= G * (HD / 2) && idx < kPairs) {
                    const bool is_k = idx < (G + 1) * (HD / 2);
                    *reinterpret_cast<uint32_t *>(is_k ? &sm.tile.k[buf][pos - t0][2 * i] : &sm.tile.v[buf][pos - t0][2 * i]) = fresh[r];
                }
            }
            __syncthreads();
        }
        const int key0 = 16 * kg;
        if (t0 + key0 >= end) continue;
        // Every product has an accumulator of its own and is added by the rounding adder, pairs of pairs: the tensor core cuts
        // additions off.
        float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f}, level[2][8];
        const uint32_t qa = smem_u32(&sm.q[0][0]) + uint32_t((lane & 15) * LD + (lane >> 4) * 8) * 2;
        const uint32_t ka = k0 + uint32_t((buf * kTile + key0 + (lane & 7) + ((lane >> 4) & 1) * 8) * LD + ((lane >> 3) & 1) * 8) * 2;
#pragma unroll
        for (int ks = 0; ks < HD / 16; ++ks) {
            uint32_t qf[4], kf[4];
            ldmatrix4(qf, qa + ks * 32);
            ldmatrix4(kf, ka + ks * 32);
            float x0[4] = {0.f, 0.f, 0.f, 0.f}, x1[4] = {0.f, 0.f, 0.f, 0.f};
            mma_f16(x0, qf, kf[0], kf[1]);
            mma_f16(x1, qf, kf[2], kf[3]);
            if constexpr (QT == 2) {  // the third parts, rows 0-7 of the second tile
                uint32_t ql[4];
                float y0[4] = {0.f, 0.f, 0.f, 0.f}, y1[4] = {0.f, 0.f, 0.f, 0.f};
                ldmatrix4(ql, qa + uint32_t(16 * LD * 2) + ks * 32);
                mma_f16(y0, ql, kf[0], kf[1]);
                mma_f16(y1, ql, kf[2], kf[3]);
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    x0[2 + e] += y0[e];
                    x1[2 + e] += y1[e];
                }
            }
            // x = the sum of a whole block of 2^n steps: up the tree as long as its partner waits there
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float x = x0[e], y = x1[e];
                if ((ks & 1) != 0) {
                    x += level[0][e];
                    y += level[0][4 + e];
                    if ((ks & 2) != 0) {
                        s0[e] += x + level[1][e];
                        s1[e] += y + level[1][4 + e];
                    } else {
                        level[1][e] = x;
                        level[1][4 + e] = y;
                    }
                } else {
                    level[0][e] = x;
                    level[0][4 + e] = y;
                }
            }
        }
        // this lane: head gl % G against keys 2t, 2t + 1 of either eight
        float s[4] = {join(s0[0] + s0[2]), join(s0[1] + s0[3]), join(s1[0] + s1[2]), join(s1[1] + s1[3])};
        float top = -INFINITY;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int key = t0 + key0 + (c >> 1) * 8 + 2 * t + (c & 1);
            s[c] = key < end ? s[c] * to_score : -INFINITY;
            top = fmaxf(top, s[c]);
        }
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
        const float mn = fmaxf(m, top);
        // a score of -inf (an infinite key, or a masked one) has no weight, also when there is no larger one yet; NaN stays
        const float corr = mn == -INFINITY ? 1.0f : expf(m - mn);
        m = mn;
        uint32_t pf[QT][4];
        __half part[4][3];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            s[c] = s[c] == -INFINITY ? 0.f : expf(s[c] - mn);
            split3(s[c] * kUp, part[c]);
        }
        l = fmaf(l, corr, (s[0] + s[1]) + (s[2] + s[3]));
        // rows gl and gl + 8 of the probability tile(s), laid out as the queries'
#pragma unroll
        for (int f = 0; f < 2; ++f) {
            uint32_t w[3];
#pragma unroll
            for (int p = 0; p < 3; ++p) {
                const __half2 h = __halves2half2(part[2 * f][p], part[2 * f + 1][p]);
                w[p] = *reinterpret_cast<const uint32_t *>(&h);
            }
            const int which = gl / G;
            if constexpr (G == 8) {
                pf[0][2 * f] = w[0];
                pf[0][2 * f + 1] = w[1];
                pf[QT - 1][2 * f] = w[2];
                pf[QT - 1][2 * f + 1] = 0u;
            } else {
                pf[0][2 * f] = which == 0 ? w[0] : which == 1 ? w[1] : 0u;
                pf[0][2 * f + 1] = which == 1 ? w[2] : 0u;
            }
        }
        const uint32_t va = v0 + uint32_t((buf * kTile + key0 + (lane & 15)) * LD + half * (HD / 2) + (lane >> 4) * 8) * 2;
#pragma unroll
        for (int d = 0; d < DB; d += 2) {
            uint32_t vf[4];
            ldmatrix4_trans(vf, va + d * 16);
            float x0[4] = {0.f, 0.f, 0.f, 0.f}, x1[4] = {0.f, 0.f, 0.f, 0.f};
            if constexpr (QT == 2) {
                mma_f16(x0, pf[1], vf[0], vf[1]);
                mma_f16(x1, pf[1], vf[2], vf[3]);
            }
            mma_f16(x0, pf[0], vf[0], vf[1]);
            mma_f16(x1, pf[0], vf[2], vf[3]);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                o[d][e] = fmaf(o[d][e], corr, x0[e]);
                o[d + 1][e] = fmaf(o[d + 1][e], corr, x1[e]);
            }
        }
    }
    trace_mark(trace, 4);
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);
    __syncthreads();  // everybody is done with the tiles: their memory becomes the merge area
    float all[2] = {0.f, 0.f};  // sums of this thread's outputs: infinite or NaN when one is
#pragma unroll
    for (int d = 0; d < DB; ++d) {
        const float x = join(o[d][0] + o[d][2]), y = join(o[d][1] + o[d][3]);
        all[0] += x;
        all[1] += y;
        if (gl < G) {
            sm.merge[kg][gl][half * (HD / 2) + d * 8 + 2 * t] = x * (1.0f / kUp);
            sm.merge[kg][gl][half * (HD / 2) + d * 8 + 2 * t + 1] = y * (1.0f / kUp);
        }
    }
    if (half == 0 && gl < G && t == 0) {
        sm.merge[kg][gl][HD] = m;
        sm.merge[kg][gl][HD + 1] = l;
    }
    // (a NaN score makes all outputs of its head NaN, so that they show it)
    if (__builtin_expect(__syncthreads_or(!(fabsf(all[0] + all[1]) < INFINITY)), 0)) {
        scalar_range<HD, G>(a, sm);
        __syncthreads();
    }
    if (tid < G * kGroups) {  // four lanes per head: the groups' maxima and sums (one without keys weighs nothing)
        const int g = tid / kGroups, w = tid % kGroups;
        const unsigned lanes = G * kGroups >= 32 ? 0xffffffffu : (1u << (G * kGroups)) - 1u;
        const float mw = sm.merge[w][g][HD];
        float M = mw;
#pragma unroll
        for (int s = 1; s < kGroups; s *= 2) M = fmaxf(M, __shfl_xor_sync(lanes, M, s));
        const float wgt = mw == -INFINITY ? 0.f : expf(mw - M);
        float L = sm.merge[w][g][HD + 1] * wgt;
#pragma unroll
        for (int s = 1; s < kGroups; s *= 2) L += __shfl_xor_sync(lanes, L, s);
        sm.w[w][g] = wgt;
        if (w == 0) {
            sm.top[g] = M;
            sm.sum[g] = L;
        }
    }
    __syncthreads();
    float *parts = a.partial + (size_t(b) * a.kv_heads + kvh) * a.nsplit * (G * ROW);  // [range][head][HD + 2]
    for (int idx = tid; idx < G * HD; idx += kThreads) {
        const int g = idx / HD, d = idx - g * HD;
        float part[kGroups];
#pragma unroll
        for (int w = 0; w < kGroups; ++w) part[w] = sm.merge[w][g][d] * sm.w[w][g];
        const float val = sum_pairs(part);
        if (nsplit == 1) {
            attn_store(a, size_t(b), (kvh * G + g) * HD + d, val / sm.sum[g]);
        } else {
            float *p = parts + (size_t(split) * G + g) * ROW;
            p[d] = val;
            if (d == 0) {
                p[HD] = sm.top[g];
                p[HD + 1] = sm.sum[g];
            }
        }
    }
    if (nsplit == 1) {
        trace_mark(trace, 5);
        if (tid == 0) trace_cta_exit();
        return;
    }
    // The last range of this (row, KV head) to finish folds them all.
    __syncthreads();
    unsigned *arrived = a.counters + size_t(b) * a.kv_heads + kvh;
    if (tid == 0) {
        unsigned before;
        asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(before) : "l"(arrived) : "memory");
        sm.is_last = before == unsigned(nsplit) - 1u;
    }
    __syncthreads();
    if (!sm.is_last) return;
    for (int idx = tid; idx < G * nsplit; idx += kThreads) sm.fold[idx] = __ldcg(parts + size_t(idx) * ROW + HD);  // [range][head]
    // this thread's output elements in the first ranges, on their way meanwhile
    auto weighted_pairs = [](const auto &x, const float *w) {  // the sum of x[i] w[i G]
        constexpr int N = sizeof(x) / sizeof(float);
        float s[N / 2];
#pragma unroll
        for (int i = 0; i < N / 2; ++i) s[i] = fmaf(x[2 * i + 1], w[(2 * i + 1) * G], x[2 * i] * w[2 * i * G]);
        return sum_pairs(s);
    };
    constexpr int kOut = (G * HD + kThreads - 1) / kThreads, kEarly = 4;
    float mine[kOut][kEarly];
#pragma unroll
    for (int r = 0; r < kOut; ++r) {
        const int idx = tid + r * kThreads;
#pragma unroll
        for (int s = 0; s < kEarly; ++s) mine[r][s] = idx < G * HD && s < nsplit ? __ldcg(parts + (size_t(s) * G + idx / HD) * ROW + idx % HD) : 0.f;
    }
    __syncthreads();
    if (warp < G) {
        // no weight for what fills up the first batch of loads, or the last one
        if (lane < 12) sm.fold[(nsplit + lane) * G + warp] = 0.f;
        float M = -INFINITY;
        for (int s = lane; s < nsplit; s += 32) M = fmaxf(M, sm.fold[s * G + warp]);
        M = warp_max(M);
        float L = 0.f;
        for (int s = lane; s < nsplit; s += 32) {
            const float ms = sm.fold[s * G + warp];
            const float w = ms == -INFINITY ? 0.f : expf(ms - M);
            sm.fold[s * G + warp] = w;
            L += __ldcg(parts + (size_t(s) * G + warp) * ROW + HD + 1) * w;
        }
        L = warp_sum(L);
        if (lane == 0) sm.inv[warp] = 1.0f / L;
    }
    __syncthreads();
    float val[kOut];
#pragma unroll
    for (int r = 0; r < kOut; ++r) val[r] = weighted_pairs(mine[r], &sm.fold[(tid + r * kThreads) / HD % G]);
    for (int s0 = kEarly; s0 < nsplit; s0 += 8) {
        float more[kOut][8];  // eight ranges of all of this thread's elements in flight
#pragma unroll
        for (int r = 0; r < kOut; ++r) {
            const int idx = tid + r * kThreads;
#pragma unroll
            for (int s = 0; s < 8; ++s) more[r][s] = idx < G * HD && s0 + s < nsplit ? __ldcg(parts + (size_t(s0 + s) * G + idx / HD) * ROW + idx % HD) : 0.f;
        }
#pragma unroll
        for (int r = 0; r < kOut; ++r) val[r] += weighted_pairs(more[r], &sm.fold[s0 * G + (tid + r * kThreads) / HD % G]);
    }
#pragma unroll
    for (int r = 0; r < kOut; ++r) {
        const int idx = tid + r * kThreads;
        if (idx < G * HD) attn_store(a, size_t(b), kvh * (G * HD) + idx, val[r] * sm.inv[idx / HD]);
    }
    if (tid == 0) {
        *arrived = 0u;
        trace_cta_exit();
    }
    trace_mark(trace, 5);
}

template <int HD, int G>
cudaError_t launch_t(const AttnArgs &a, int width, cudaStream_t stream, bool programmatic) {
    static_assert((kAttnMaxSplits + 12) * G <= 1024, "the fold's table");
    if (a.nsplit < 1 || a.nsplit > kAttnMaxSplits) return cudaErrorInvalidValue;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(a.nsplit, a.kv_heads, width);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = sizeof(typename SplitAttn<HD, G>::Smem);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = programmatic ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, attn_split_kernel<HD, G>, a);
}
template <int HD>
cudaError_t launch_hd(const AttnArgs &a, int width, cudaStream_t stream, bool programmatic) {
    switch (a.heads / a.kv_heads) {
        case 1: return launch_t<HD, 1>(a, width, stream, programmatic);
        case 2: return launch_t<HD, 2>(a, width, stream, programmatic);
        case 4: return launch_t<HD, 4>(a, width, stream, programmatic);
        case 8: return launch_t<HD, 8>(a, width, stream, programmatic);
        default: return cudaErrorInvalidValue;
    }
}
template <int HD, int G>
cudaError_t configure_t() {
    return cudaFuncSetAttribute(attn_split_kernel<HD, G>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(typename SplitAttn<HD, G>::Smem)));
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

cudaError_t attention_split_configure() {
    const cudaError_t e = configure_hd<128>();
    return e != cudaSuccess ? e : configure_hd<64>();
}

cudaError_t attention_launch(const AttnArgs &a, int width, cudaStream_t stream, bool programmatic) {
    if (a.head_dim == 128) return launch_hd<128>(a, width, stream, programmatic);
    if (a.head_dim == 64) return launch_hd<64>(a, width, stream, programmatic);
    return cudaErrorInvalidValue;
}

}  // namespace jl
