// Per-layer kernels around the matrix products (see ops.cuh).
#include "ops.cuh"

#include <cuda_fp16.h>

#include <algorithm>

namespace jl {

JL_TRACE_DEFINE_BIND(ops_trace_bind)

namespace {

// ---- embedding -------------------------------------------------------------------------------
__global__ void embedding_kernel(int type, const uint8_t *table, const int32_t *tokens,
                                 const uint8_t *active, float *x, int dim) {
    const int row = blockIdx.y;
    const bool on = active == nullptr || active[row] != 0;
    pdl_wait();
    pdl_launch_dependents();
    if (!on) return;
    const int token = tokens[row];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < dim; i += gridDim.x * blockDim.x)
        x[size_t(row) * dim + i] = decode_any(type, table, int64_t(token) * dim + i);
}

// ---- dequant ---------------------------------------------------------------------------------
__global__ void dequant_kernel(int type, const uint8_t *blocks, int64_t n, float *out) {
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride)
        out[i] = decode_any(type, blocks, i);
}

// Q6_K super-blocks (210 bytes) copied into slots of kQ6_KPadded bytes, the tail zeroed: the layout the tensor-core
// kernel's 2-D tensor map needs (rows that are 16-byte multiples). 16-bit pieces: the source is 2-byte aligned.
__global__ void pad_q6k_kernel(const uint8_t *src, uint8_t *dst, size_t nblocks) {
    constexpr int kHalfWords = kQ6_KPadded / 2;
    const size_t total = nblocks * kHalfWords, stride = size_t(gridDim.x) * blockDim.x;
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += stride) {
        const size_t blk = i / kHalfWords;
        const int w = int(i - blk * kHalfWords);
        const unsigned short v = w < kQ6_KBytes / 2 ? reinterpret_cast<const unsigned short *>(src + blk * kQ6_KBytes)[w] : 0;
        reinterpret_cast<unsigned short *>(dst + blk * kQ6_KPadded)[w] = v;
    }
}

__global__ void fill_kernel(uint32_t *buf, size_t words, uint32_t value) {
    const size_t stride = size_t(gridDim.x) * blockDim.x;
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < words; i += stride)
        buf[i] = value;
}

__global__ void advance_kernel(int32_t *tokens, int32_t *positions, const int32_t *sampled,
                               const uint8_t *active, int32_t *history, int32_t *step_counter,
                               int width) {
    pdl_wait();
    pdl_launch_dependents();
    const int b = threadIdx.x;
    const int step = *step_counter;
    __syncthreads();
    if (b < width) {
        const bool on = active[b] != 0;
        const int32_t tok = on ? sampled[b] : -1;
        history[size_t(step) * width + b] = tok;
        if (on) {
            tokens[b] = tok;
            positions[b] += 1;
        }
    }
    if (b == 0) *step_counter = step + 1;
}

__device__ __forceinline__ int64_t kv_offset(const KvGeom &g, int slot, int pos, int layer) {
    const int blk = pos / g.block_tokens;
    const int within = pos - blk * g.block_tokens;
    const int64_t phys = g.block_table[int64_t(slot) * g.blocks_per_slot + blk];
    const int64_t block_stride = int64_t(g.layers) * g.block_tokens * g.kv_dim;
    return phys * block_stride + int64_t(layer) * g.block_tokens * g.kv_dim +
           int64_t(within) * g.kv_dim;
}

// The row kernels below take part in chains of programmatic dependent launches: each lets the next
// kernel start its preamble at once (a matrix-matrix kernel then streams its first weights while this
// one runs) and waits for the kernel before it. Every CTA waits, also one that then has nothing to do:
// a grid whose CTAs left without waiting would count as complete while its predecessor still runs,
// and the next kernel's wait covers only its own predecessor. The embedding and the advance kernel
// wait before they release: whatever starts after them may read the step's positions at once.
__global__ void add_rows_kernel(float *x, const float *y, size_t total) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t stride = size_t(gridDim.x) * blockDim.x;
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += stride) x[i] = x[i] + y[i];
}

// Four consecutive activations as binary16 hi and lo parts (x = hi + lo), the tensor-core path's
// activation format. Inside each group of four the pairs are (x0, x2) and (x1, x3): the weight
// conversion gets the nibbles of bytes 0 and 2 of a word with one logic operation, and a sum over K
// does not care about the order as long as both operands use the same one.
__device__ __forceinline__ void split4_store(const float4 v, uint2 *hi, uint2 *lo) {
    const __half2 h0 = __floats2half2_rn(v.x, v.z), h1 = __floats2half2_rn(v.y, v.w);
    const float2 b0 = __half22float2(h0), b1 = __half22float2(h1);
    const __half2 l0 = __floats2half2_rn(v.x - b0.x, v.z - b0.y), l1 = __floats2half2_rn(v.y - b1.x, v.w - b1.y);
    *hi = make_uint2(*reinterpret_cast<const uint32_t *>(&h0), *reinterpret_cast<const uint32_t *>(&h1));
    *lo = make_uint2(*reinterpret_cast<const uint32_t *>(&l0), *reinterpret_cast<const uint32_t *>(&l1));
}

__global__ void split_rows_kernel(const float4 *x, size_t total4, uint2 *hi, uint2 *lo) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t stride = size_t(gridDim.x) * blockDim.x;
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < total4; i += stride) {
        split4_store(x[i], hi + i, lo + i);
    }
}

__global__ void tp_pack_best_kernel(const float *logits, const int32_t *idx, int l_vocab, int index_offset, int n,
                                    float *best) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    const int i = idx[r];
    best[2 * r] = logits[size_t(r) * l_vocab + i];
    best[2 * r + 1] = static_cast<float>(i + index_offset);  // vocabulary indices are exact in fp32
}

__global__ void tp_pick_best_kernel(const float *all, int ranks, int n, const uint8_t *active, int32_t *out) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n || (active != nullptr && active[r] == 0)) return;
    float bv = -INFINITY;
    int bi = 0x7fffffff;
    for (int k = 0; k < ranks; ++k) {
        const float v = all[(size_t(k) * n + r) * 2];
        const int i = static_cast<int>(all[(size_t(k) * n + r) * 2 + 1]);
        if (v > bv || (v == bv && i < bi)) {
            bv = v;
            bi = i;
        }
    }
    out[r] = bi == 0x7fffffff ? 0 : bi;
}

// ---- row-wise operators for the matrix-matrix path ---------------------------------------------
// One CTA per row. The row is read once, as float4 batches held in registers (all loads issued
// before the first use: one L2 round trip, not one per element), and the same registers feed the
// output pass. The norm's weights, which no kernel writes, are in flight while the kernel ahead still runs: loaded after
// the sum they cost a second round trip, to memory (65 such launches in a step of 32 rows: 4192 -> 4110 us).
// Optionally also writes the row as binary16 hi / lo parts (x = hi + lo), the activation format of the
// tensor-core path.
constexpr int kNormThreads = 256;
constexpr int kNormBatch = 8;  // float4 per thread per batch: rows up to 8192 in one batch

__global__ void __launch_bounds__(kNormThreads) rmsnorm_rows_kernel(const float *x, const float *w, float eps, float *out,
                                                                    int dim, const uint8_t *active, uint2 *hi, uint2 *lo) {
    const int row = blockIdx.x;
    const int trace = trace_begin(kTraceRows);
    trace_word(trace, 7, 1);
    pdl_launch_dependents();
    __shared__ float part[9];
    const int n4 = dim / 4;
    const float4 *xr = reinterpret_cast<const float4 *>(x + size_t(row) * dim);
    const float4 *w4 = reinterpret_cast<const float4 *>(w);
    float4 v[kNormBatch], g[kNormBatch];
#pragma unroll
    for (int k = 0; k < kNormBatch; ++k) {
        const int i = k * kNormThreads + threadIdx.x;
        g[k] = i < n4 ? w4[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    pdl_wait();
    if (active != nullptr && active[row] == 0) return;
#pragma unroll
    for (int k = 0; k < kNormBatch; ++k) {
        const int i = k * kNormThreads + threadIdx.x;
        v[k] = i < n4 ? xr[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < kNormBatch; ++k) s += v[k].x * v[k].x + v[k].y * v[k].y + v[k].z * v[k].z + v[k].w * v[k].w;
    for (int i = kNormBatch * kNormThreads + threadIdx.x; i < n4; i += kNormThreads) {
        const float4 u = xr[i];
        s += u.x * u.x + u.y * u.y + u.z * u.z + u.w * u.w;
    }
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        float tot = 0.f;
        for (int i = 0; i < kNormThreads / 32; ++i) tot += part[i];
        float ms = tot / static_cast<float>(dim);
        ms += eps;
        part[8] = static_cast<float>(1.0 / sqrt(static_cast<double>(ms)));
    }
    __syncthreads();
    const float ss = part[8];
    float4 *o4 = reinterpret_cast<float4 *>(out + size_t(row) * dim);
    uint2 *hr = hi != nullptr ? hi + size_t(row) * n4 : nullptr;
    uint2 *lr = lo != nullptr ? lo + size_t(row) * n4 : nullptr;
    auto emit = [&](int i, float4 u, float4 g) {
        float4 r;
        r.x = __fmul_rn(g.x, __fmul_rn(ss, u.x));
        r.y = __fmul_rn(g.y, __fmul_rn(ss, u.y));
        r.z = __fmul_rn(g.z, __fmul_rn(ss, u.z));
        r.w = __fmul_rn(g.w, __fmul_rn(ss, u.w));
        o4[i] = r;
        if (hr != nullptr) split4_store(r, hr + i, lr + i);
    };
#pragma unroll
    for (int k = 0; k < kNormBatch; ++k) {
        const int i = k * kNormThreads + threadIdx.x;
        if (i < n4) emit(i, v[k], g[k]);
    }
    for (int i = kNormBatch * kNormThreads + threadIdx.x; i < n4; i += kNormThreads) emit(i, xr[i], w4[i]);
}

// Four elements per thread per step (row lengths are multiples of 256, so float4 never straddles).
__global__ void swiglu_rows_kernel(float4 *g, const float4 *u, size_t total4, uint2 *hi, uint2 *lo) {
    const int trace = trace_begin(kTraceRows);
    trace_word(trace, 7, 2);
    pdl_launch_dependents();
    pdl_wait();
    const size_t stride = size_t(gridDim.x) * blockDim.x;
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < total4; i += stride) {
        const float4 v = g[i], w = u[i];
        float4 r;
        r.x = (v.x / (1.0f + expf(-v.x))) * w.x;
        r.y = (v.y / (1.0f + expf(-v.y))) * w.y;
        r.z = (v.z / (1.0f + expf(-v.z))) * w.z;
        r.w = (v.w / (1.0f + expf(-v.w))) * w.w;
        g[i] = r;
        if (hi != nullptr) split4_store(r, hi + i, lo + i);
    }
}

__global__ void kv_append_kernel(const float *k, const float *v, const float *rope_cos, const float *rope_sin,
                                 const int32_t *positions, const int32_t *slots, const uint8_t *active,
                                 KvGeom kv, int layer, int head_dim) {
    const int row = blockIdx.x;
    pdl_launch_dependents();
    pdl_wait();
    if (active != nullptr && active[row] == 0) return;
    const int pos = positions[row], slot = slots[row];
    const int64_t off = kv_offset(kv, slot, pos, layer);
    const float *kr = k + size_t(row) * kv.kv_dim, *vr = v + size_t(row) * kv.kv_dim;
    const int half = head_dim / 2;
    for (int p = threadIdx.x; p < kv.kv_dim / 2; p += blockDim.x) {
        const int i = p % half;
        const float cr = rope_cos[size_t(pos) * half + i], ci = rope_sin[size_t(pos) * half + i];
        const float v0 = kr[2 * p], v1 = kr[2 * p + 1];
        kv.kpool[off + 2 * p] = __float2half_rn(__fsub_rn(__fmul_rn(v0, cr), __fmul_rn(v1, ci)));
        kv.kpool[off + 2 * p + 1] = __float2half_rn(__fadd_rn(__fmul_rn(v0, ci), __fmul_rn(v1, cr)));
        kv.vpool[off + 2 * p] = __float2half_rn(vr[2 * p]);
        kv.vpool[off + 2 * p + 1] = __float2half_rn(vr[2 * p + 1]);
    }
}

// The first index of each row's maximum, one CTA of 1024 threads per row. A row of 128 256 logits is 513 KB and sits in
// L2 (the projection just wrote it), so the kernel is bound by the loads a CTA keeps in flight: with 4-byte loads
// issued between the comparisons, 126 to a thread, it was a chain of round trips; eight 16-byte loads in flight leave
// four of them (a step of 32 rows 4540 -> 4519 us). Rows that do not start on 16 bytes (a vocabulary that is no
// multiple of 4) take eight 4-byte loads instead.
constexpr int kArgmaxLoads = 8;

__global__ void __launch_bounds__(1024) argmax_rows_kernel(const float *logits, int vocab, const uint8_t *active,
                                                           int32_t *out) {
    const int row = blockIdx.x;
    pdl_launch_dependents();
    pdl_wait();
    if (active != nullptr && active[row] == 0) return;
    const float *lr = logits + size_t(row) * vocab;
    float bv = -INFINITY;
    int bi = 0x7fffffff;
    auto take = [&](float v, int i) {  // a thread visits its indices in increasing order: ties go to the first
        if (v > bv) {
            bv = v;
            bi = i;
        }
    };
    const int step = int(blockDim.x);
    if ((vocab & 3) == 0 && (reinterpret_cast<uintptr_t>(logits) & 15) == 0) {
        const float4 *lr4 = reinterpret_cast<const float4 *>(lr);
        const int n4 = vocab >> 2;
        for (int base = threadIdx.x; base < n4; base += step * kArgmaxLoads) {
            float4 q[kArgmaxLoads];
#pragma unroll
            for (int u = 0; u < kArgmaxLoads; ++u)
                q[u] = base + u * step < n4 ? lr4[base + u * step]
                                            : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
#pragma unroll
            for (int u = 0; u < kArgmaxLoads; ++u) {
                const int i = 4 * (base + u * step);
                take(q[u].x, i);
                take(q[u].y, i + 1);
                take(q[u].z, i + 2);
                take(q[u].w, i + 3);
            }
        }
    } else {
        for (int base = threadIdx.x; base < vocab; base += step * kArgmaxLoads) {
            float q[kArgmaxLoads];
#pragma unroll
            for (int u = 0; u < kArgmaxLoads; ++u) q[u] = base + u * step < vocab ? lr[base + u * step] : -INFINITY;
#pragma unroll
            for (int u = 0; u < kArgmaxLoads; ++u) take(q[u], base + u * step);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > bv || (ov == bv && oi < bi)) {
            bv = ov;
            bi = oi;
        }
    }
    __shared__ float sv[32];
    __shared__ int si[32];
    if ((threadIdx.x & 31) == 0) {
        sv[threadIdx.x >> 5] = bv;
        si[threadIdx.x >> 5] = bi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < int(blockDim.x >> 5); ++w)
            if (sv[w] > bv || (sv[w] == bv && si[w] < bi)) {
                bv = sv[w];
                bi = si[w];
            }
        out[row] = bi == 0x7fffffff ? 0 : bi;
    }
}

__device__ __forceinline__ void cp_async_16(uint32_t dst_smem, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst_smem), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

__device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// ---- decode attention for wide batches: the query heads of a KV head as the rows of an MMA tile ---------------
// One CTA per (batch row, KV head). The G query heads that share the KV head are rows 0..G-1 of the 16-row A
// operand (the other rows are zero), so the scores of all heads against 64 keys are 16 mma.sync per key tile
// and warp instead of a few thousand scalar multiply-adds, and the kernel runs at the speed the pages arrive.
// The four warps are independent until the end: of every 64 keys each takes sixteen, stages them in a ring of its
// own (cp.async, two groups of sixteen ahead) and keeps its own running maximum, sum and output, merged at the end.
// Nothing but the pages' arrival should bound this kernel, so the instructions beside the products are few: the
// sixteen keys of a group share a page whenever the page size is a multiple of sixteen, and then one page lookup and
// one pointer serve all of a lane's copies of the group; no barrier of the CTA stands between two groups. A step of the 8B
// shape with 32 rows of 256-768 keys takes 4210 us this way; with tiles of 64 keys staged by the whole CTA, an address division
// for every key and two barriers a tile it is 4519 (9.7 us more in each of 32 launches).
// The step's own key and value (rotated, rounded to binary16 as the append does) are written to the page and
// dropped into the staged group by the warp that holds it, so nothing else has to run before it.
// Arithmetic: inference/op/CpuOperations.java:94-235, as attn_split.cu.
template <int HD, int G>
struct BatchAttnShape {
    static constexpr int warps = 4;
    static constexpr int tk = 16;       // keys per group, the depth of one MMA of the value product
    static constexpr int depth = 3;     // group buffers per warp: two groups in flight while one is used
    static constexpr int ld = HD + 8;
    static constexpr int pages = 256;   // page bases kept in shared memory (4 K keys of 16-token pages)
    static constexpr int tile_halves = tk * ld;
    static constexpr int merge_floats = warps * G * (HD + 2);  // overlays the tiles once the keys are done
    static constexpr int ring_bytes = warps * depth * 2 * tile_halves * 2;
    static constexpr int smem_bytes = ring_bytes + pages * 8;  // two CTAs per SM at HD = 128
    static_assert(merge_floats * 4 <= ring_bytes, "the merge area overlays the rings");
};

template <int HD, int G>
__global__ void __launch_bounds__(BatchAttnShape<HD, G>::warps * 32, 2)
    attn_batch_kernel(const AttnArgs a) {
    using P = BatchAttnShape<HD, G>;
    constexpr int TK = P::tk, LD = P::ld, KS = HD / 16, DB = HD / 8, NBUF = P::depth;
    constexpr int PARTS = HD / 8;               // 16-byte chunks per key row
    constexpr int KEYS_PER_PASS = 32 / PARTS;   // key rows one pass of a warp's lanes covers
    extern __shared__ __align__(16) uint8_t batch_smem[];
    int64_t *page_base = reinterpret_cast<int64_t *>(batch_smem + P::ring_bytes);
    float *merge = reinterpret_cast<float *>(batch_smem);  // after the last group
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    __half *ring = reinterpret_cast<__half *>(batch_smem) + warp * NBUF * 2 * P::tile_halves;  // [buffer][K | V][TK][LD]
    const int kvh = blockIdx.x, b = blockIdx.y;
    const int qr = lane >> 2, qc = lane & 3;
    const bool on = a.active == nullptr || a.active[b] != 0;
    const int trace = trace_begin(kTraceAttn);
    pdl_launch_dependents();
    // positions, slots and the block table are not written by anything in this step (see attn_split.cu)
    const int pos = on ? a.positions[b] : -1;
    const int slot = on ? a.slots[b] : 0;
    const int bt = a.kv.block_tokens;
    if (on) {
        const int64_t block_stride = int64_t(a.kv.layers) * bt * a.kv.kv_dim;
        for (int pg = tid; pg < min(pos / bt + 1, P::pages); pg += P::warps * 32) {
            const int64_t phys = a.kv.block_table[int64_t(slot) * a.kv.blocks_per_slot + pg];
            page_base[pg] = phys * block_stride + int64_t(a.layer) * bt * a.kv.kv_dim + int64_t(kvh) * HD;
        }
    }
    __syncthreads();
    const uint32_t ring_u32 = static_cast<uint32_t>(__cvta_generic_to_shared(ring));
    auto key_offset = [&](int t) -> int64_t {
        const int pg = t / bt;
        const int64_t base = pg < P::pages ? page_base[pg] : kv_offset(a.kv, slot, t - t % bt, a.layer) + int64_t(kvh) * HD;
        return base + int64_t(t % bt) * a.kv.kv_dim;
    };
    // Group g of this warp: keys first_key + 64 g .. + 15. Keys 0 .. pos - 1 come from the pages (this step's key,
    // position pos, is written below); a lane copies the same 16-byte part of every KEYS_PER_PASS-th key row.
    constexpr int STRIDE = P::warps * TK;
    const int first_key = warp * TK;
    const int part = lane % PARTS, key_first = lane / PARTS;
    const bool one_page = bt % TK == 0;  // the sixteen keys of every group lie in one page
    auto stage = [&](int g, int buf) {
        const int t0 = first_key + g * STRIDE;
        const uint32_t dst = ring_u32 + uint32_t(((buf * 2) * P::tile_halves + key_first * LD + part * 8) * 2);
        constexpr uint32_t V = uint32_t(P::tile_halves * 2);
        if (one_page && t0 + TK <= pos) {
            const int64_t off = key_offset(t0) + int64_t(key_first) * a.kv.kv_dim + part * 8;
            const __half *ks = a.kv.kpool + off, *vs = a.kv.vpool + off;
            const int step = KEYS_PER_PASS * a.kv.kv_dim;
#pragma unroll
            for (int i = 0; i < TK / KEYS_PER_PASS; ++i) {
                cp_async_16(dst + uint32_t(i * KEYS_PER_PASS * LD * 2), ks);
                cp_async_16(dst + V + uint32_t(i * KEYS_PER_PASS * LD * 2), vs);
                ks += step;
                vs += step;
            }
        } else {  // a page size that is no multiple of sixteen, or the last keys
#pragma unroll 1
            for (int i = 0; i < TK / KEYS_PER_PASS; ++i) {
                const uint32_t dk = dst + uint32_t(i * KEYS_PER_PASS * LD * 2);
                const int t = t0 + key_first + i * KEYS_PER_PASS;
                if (t < pos) {
                    const int64_t off = key_offset(t) + part * 8;
                    cp_async_16(dk, a.kv.kpool + off);
                    cp_async_16(dk + V, a.kv.vpool + off);
                } else {
                    asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(dk), "r"(0u) : "memory");
                    asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(dk + V), "r"(0u) : "memory");
                }
            }
        }
        cp_async_commit();
    };
    const int ngroups = pos >= first_key ? (pos - first_key) / STRIDE + 1 : 0;  // none when the row is off
    // old keys: in flight while the kernel ahead finishes (one commit group per ring slot, empty ones included,
    // so that "all but the newest NBUF - 2 groups" always means "the group about to be used")
#pragma unroll
    for (int p = 0; p < NBUF - 1; ++p) {
        if (p < ngroups) stage(p, p);
        else cp_async_commit();
    }
    pdl_wait();
    trace_mark(trace, 2);
    if (!on) return;
    // The G heads' queries, rotated, as rows 0..G-1 of the A operand (hi and lo binary16 parts); rows G..15 are zero.
    uint32_t qhi[KS][2], qlo[KS][2];  // a0 and a2 of each K step: a1 / a3 (rows 8..15) are zero
    const float *cr = a.rope_cos + size_t(pos) * (HD / 2), *ci = a.rope_sin + size_t(pos) * (HD / 2);
#pragma unroll
    for (int k = 0; k < KS; ++k) {
#pragma unroll
        for (int f = 0; f < 2; ++f) {
            const int d0 = 16 * k + 8 * f + 2 * qc;
            float x0 = 0.f, x1 = 0.f;
            if (qr < G) {
                const float *qh = a.q + size_t(b) * a.dim + size_t(kvh * G + qr) * HD;
                const float v0 = qh[d0], v1 = qh[d0 + 1];
                x0 = __fsub_rn(__fmul_rn(v0, cr[d0 / 2]), __fmul_rn(v1, ci[d0 / 2]));
                x1 = __fadd_rn(__fmul_rn(v0, ci[d0 / 2]), __fmul_rn(v1, cr[d0 / 2]));
            }
            const __half2 hi = __floats2half2_rn(x0, x1);
            const float2 back = __half22float2(hi);
            const __half2 lo = __floats2half2_rn(x0 - back.x, x1 - back.y);
            qhi[k][f] = *reinterpret_cast<const uint32_t *>(&hi);
            qlo[k][f] = *reinterpret_cast<const uint32_t *>(&lo);
        }
    }
    float o[DB][4];
#pragma unroll
    for (int db = 0; db < DB; ++db) o[db][0] = o[db][1] = o[db][2] = o[db][3] = 0.f;
    float m = -INFINITY, l = 0.f;  // of row qr (a head when qr < G)
    const float inv_sqrt = 1.0f / sqrtf(static_cast<float>(HD));
    trace_mark(trace, 3);
    // ldmatrix rows of this lane: keys (lane & 7) and + 8 for the upper two of a K x4, 8 dims further for the odd ones;
    // keys (lane & 15) of the values, 8 dims further for the upper half of the lanes
    const uint32_t k_lane = uint32_t((((lane & 7) + ((lane >> 4) << 3)) * LD + ((lane >> 3) & 1) * 8) * 2);
    const uint32_t v_lane = uint32_t(((lane & 15) * LD + (lane >> 4) * 8 + P::tile_halves) * 2);
    for (int g = 0, buf = 0; g < ngroups; ++g, buf = buf + 1 == NBUF ? 0 : buf + 1) {
        const int t0 = first_key + g * STRIDE;
        asm volatile("cp.async.wait_group %0;" ::"n"(NBUF - 2) : "memory");  // this lane's copies of group g
        __syncwarp();  // every lane's copies of it have landed, and every lane is done with group g - 1
        if (g + NBUF - 1 < ngroups) stage(g + NBUF - 1, buf == 0 ? NBUF - 1 : buf - 1);  // into the buffer group g - 1 used
        else cp_async_commit();
        const uint32_t tile_u32 = ring_u32 + uint32_t(buf * 2 * P::tile_halves * 2);
        if (t0 + TK > pos) {
            // This step's key and value: rotate k, round both to binary16, into the page and into the group.
            __half *kt = ring + buf * 2 * P::tile_halves, *vt = kt + P::tile_halves;
            const int64_t off = key_offset(pos);
            const float *kh = a.k + size_t(b) * a.kv.kv_dim + size_t(kvh) * HD;
            const float *vh = a.v + size_t(b) * a.kv.kv_dim + size_t(kvh) * HD;
            for (int i = lane; i < HD / 2; i += 32) {
                const float v0 = kh[2 * i], v1 = kh[2 * i + 1];
                const __half2 hk = __halves2half2(__float2half_rn(__fsub_rn(__fmul_rn(v0, cr[i]), __fmul_rn(v1, ci[i]))),
                                                  __float2half_rn(__fadd_rn(__fmul_rn(v0, ci[i]), __fmul_rn(v1, cr[i]))));
                const __half2 hv = __halves2half2(__float2half_rn(vh[2 * i]), __float2half_rn(vh[2 * i + 1]));
                *reinterpret_cast<__half2 *>(kt + (pos - t0) * LD + 2 * i) = hk;
                *reinterpret_cast<__half2 *>(vt + (pos - t0) * LD + 2 * i) = hv;
                *reinterpret_cast<__half2 *>(a.kv.kpool + off + 2 * i) = hk;
                *reinterpret_cast<__half2 *>(a.kv.vpool + off + 2 * i) = hv;
            }
            __syncwarp();
        }
        // S = Q K^T: 16 rows (heads) x 16 keys; separate accumulators for the hi and the lo part of q, so that
        // four chains of MMAs run side by side
        float sh[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}}, sl[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
        for (int k = 0; k < KS; ++k) {
            const uint32_t ah[4] = {qhi[k][0], 0u, qhi[k][1], 0u}, al[4] = {qlo[k][0], 0u, qlo[k][1], 0u};
            uint32_t kf[2][2];  // keys 0-7 and 8-15: dims 0-7 and 8-15 of the step
            asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                         : "=r"(kf[0][0]), "=r"(kf[0][1]), "=r"(kf[1][0]), "=r"(kf[1][1])
                         : "r"(tile_u32 + k_lane + uint32_t(32 * k))
                         : "memory");
#pragma unroll
            for (int nb = 0; nb < 2; ++nb) {
                mma_16816(sh[nb], ah, kf[nb][0], kf[nb][1]);
                mma_16816(sl[nb], al, kf[nb][0], kf[nb][1]);
            }
        }
        // rows 0..7 are c0 / c1 of each lane: scale, mask the keys after pos, fold into the running soft-max
        float sv[2][2];
        float tmax = -INFINITY;
#pragma unroll
        for (int nb = 0; nb < 2; ++nb)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                sv[nb][c] = (t0 + nb * 8 + 2 * qc + c <= pos) ? (sh[nb][c] + sl[nb][c]) * inv_sqrt : -INFINITY;
                tmax = fmaxf(tmax, sv[nb][c]);
            }
        tmax = fmaxf(tmax, __shfl_xor_sync(0xffffffffu, tmax, 1));
        tmax = fmaxf(tmax, __shfl_xor_sync(0xffffffffu, tmax, 2));
        const float mn = fmaxf(m, tmax);
        const float corr = (mn == -INFINITY) ? 1.0f : expf(m - mn);
        m = mn;
        l *= corr;
        uint32_t pa[4] = {0u, 0u, 0u, 0u};  // a0 (keys 0-7) and a2 (keys 8-15) of rows 0..7; a1 / a3 (rows 8..15) stay zero
#pragma unroll
        for (int nb = 0; nb < 2; ++nb) {
            const float p0 = (m == -INFINITY) ? 0.f : expf(sv[nb][0] - m), p1 = (m == -INFINITY) ? 0.f : expf(sv[nb][1] - m);
            l += p0 + p1;
            const __half2 ph = __floats2half2_rn(p0, p1);
            pa[2 * nb] = *reinterpret_cast<const uint32_t *>(&ph);
        }
#pragma unroll
        for (int db = 0; db < DB; db += 2) {
            uint32_t vf[2][2];
            asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                         : "=r"(vf[0][0]), "=r"(vf[0][1]), "=r"(vf[1][0]), "=r"(vf[1][1])
                         : "r"(tile_u32 + v_lane + uint32_t(db * 16))
                         : "memory");
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                o[db + h][0] *= corr;
                o[db + h][1] *= corr;
                mma_16816(o[db + h], pa, vf[h][0], vf[h][1]);
            }
        }
    }
    // Merge the four warps (each saw a quarter of the keys): per head the maxima, sums and outputs.
    trace_mark(trace, 4);
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // everybody is done with the rings: their memory becomes the merge area
    if (qr < G) {
        float *mine = merge + (warp * G + qr) * (HD + 2);
#pragma unroll
        for (int db = 0; db < DB; ++db) {
            mine[db * 8 + 2 * qc] = o[db][0];
            mine[db * 8 + 2 * qc + 1] = o[db][1];
        }
        if (qc == 0) {
            mine[HD] = m;
            mine[HD + 1] = l;
        }
    }
    __syncthreads();
    for (int idx = tid; idx < G * HD; idx += P::warps * 32) {
        const int g = idx / HD, d = idx - g * HD;
        float M = -INFINITY;
#pragma unroll
        for (int w = 0; w < P::warps; ++w) M = fmaxf(M, merge[(w * G + g) * (HD + 2) + HD]);
        float val = 0.f, L = 0.f;
#pragma unroll
        for (int w = 0; w < P::warps; ++w) {
            const float *pw = merge + (w * G + g) * (HD + 2);
            const float wgt = (pw[HD] == -INFINITY) ? 0.f : expf(pw[HD] - M);
            val += pw[d] * wgt;
            L += pw[HD + 1] * wgt;
        }
        attn_store(a, size_t(b), (kvh * G + g) * HD + d, val / L);
    }
    trace_mark(trace, 5);
}

template <int HD, int G>
cudaError_t attn_batch_launch_t(const AttnArgs &a, int width, cudaStream_t stream, bool programmatic) {
    using P = BatchAttnShape<HD, G>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(a.kv_heads, width);
    cfg.blockDim = dim3(P::warps * 32);
    cfg.dynamicSmemBytes = P::smem_bytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = programmatic ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, attn_batch_kernel<HD, G>, a);
}

template <int HD>
cudaError_t attn_batch_launch_hd(const AttnArgs &a, int width, cudaStream_t s, bool pdl) {
    switch (a.heads / a.kv_heads) {
        case 1: return attn_batch_launch_t<HD, 1>(a, width, s, pdl);
        case 2: return attn_batch_launch_t<HD, 2>(a, width, s, pdl);
        case 4: return attn_batch_launch_t<HD, 4>(a, width, s, pdl);
        case 8: return attn_batch_launch_t<HD, 8>(a, width, s, pdl);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace

namespace {
template <int HD, int G>
cudaError_t attn_configure_t() {
    return cudaFuncSetAttribute(attn_batch_kernel<HD, G>, cudaFuncAttributeMaxDynamicSharedMemorySize, BatchAttnShape<HD, G>::smem_bytes);
}
template <int HD>
cudaError_t attn_configure_hd() {
    cudaError_t e;
    if ((e = attn_configure_t<HD, 1>()) != cudaSuccess) return e;
    if ((e = attn_configure_t<HD, 2>()) != cudaSuccess) return e;
    if ((e = attn_configure_t<HD, 4>()) != cudaSuccess) return e;
    return attn_configure_t<HD, 8>();
}
}  // namespace

cudaError_t attention_configure() {
    cudaError_t e;
    if ((e = attn_configure_hd<128>()) != cudaSuccess) return e;
    if ((e = attn_configure_hd<64>()) != cudaSuccess) return e;
    return attention_split_configure();
}

size_t attention_partial_floats(int width, int heads, int nsplit, int head_dim) {
    return size_t(width) * heads * nsplit * (head_dim + 2);
}

int attention_splits(int sm_count, int width, int kv_heads) {
    // Not more than two CTAs per SM over the whole launch (launches of 16 pairs or more). Below that, twenty ranges, or as many
    // as a CTA can fold in passing where few pairs would leave SMs without a CTA. A grid is sized for the longest context, and
    // CTAs that find no keys of their own cost the short ones: a step of eight layers with 8 KV heads takes 284.0 us at 57 keys with
    // 20 ranges, 285.7 with 28, 288.4 with 37 (at 8000 keys of head size 128: 539, 508, 507), five rows of one KV head (sixteen
    // layers) 687 us at 300 keys with 20 and 710 with 32. With 2 KV heads the grid stays small: 432 us at 300 keys with 20, 28 and
    // 37; 545, 521 and 510 at 4000, 891, 759 and 700 at 16000. Past 37 the fold eats the gain (48: 515 at 4000).
    const int pairs = width * kv_heads;
    return std::max(1, std::min(kAttnMaxSplits * pairs <= sm_count ? kAttnMaxSplits : 20, 2 * sm_count / pairs));
}

cudaError_t attention_batch_launch(const AttnArgs &a, int width, cudaStream_t stream, bool programmatic) {
    if (a.head_dim == 128) return attn_batch_launch_hd<128>(a, width, stream, programmatic);
    if (a.head_dim == 64) return attn_batch_launch_hd<64>(a, width, stream, programmatic);
    return cudaErrorInvalidValue;
}

cudaError_t embedding_launch(int type, const uint8_t *table, const int32_t *tokens,
                             const uint8_t *active, float *x, int dim, int width,
                             cudaStream_t stream, bool programmatic) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((dim + 255) / 256, width);
    cfg.blockDim = dim3(256);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = programmatic ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, embedding_kernel, type, table, tokens, active, x, dim);
}

cudaError_t pad_q6k_launch(const uint8_t *src, uint8_t *dst, size_t nblocks, cudaStream_t stream) {
    if (nblocks == 0) return cudaSuccess;
    const size_t want = (nblocks * (kQ6_KPadded / 2) + 255) / 256;
    pad_q6k_kernel<<<unsigned(want < 148 * 32 ? want : 148 * 32), 256, 0, stream>>>(src, dst, nblocks);
    return cudaGetLastError();
}

cudaError_t dequant_launch(int type, const uint8_t *blocks, int64_t n, float *out,
                           cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    int64_t blocks_needed = (n + 255) / 256;
    int grid = static_cast<int>(blocks_needed < 148 * 16 ? blocks_needed : 148 * 16);
    dequant_kernel<<<grid, 256, 0, stream>>>(type, blocks, n, out);
    return cudaGetLastError();
}

cudaError_t advance_launch(int32_t *tokens, int32_t *positions, const int32_t *sampled,
                           const uint8_t *active, int32_t *history, int32_t *step_counter, int width,
                           cudaStream_t stream, bool programmatic) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1);
    cfg.blockDim = dim3(256);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = programmatic ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, advance_kernel, tokens, positions, sampled, active, history,
                              step_counter, width);
}

// One launch configuration for the row kernels, with or without the programmatic-dependent-launch attribute.
struct RowLaunch {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1] = {};
    RowLaunch(int grid, int block, cudaStream_t stream, bool programmatic) {
        cfg.gridDim = dim3(unsigned(grid));
        cfg.blockDim = dim3(unsigned(block));
        cfg.stream = stream;
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = programmatic ? 1 : 0;
    }
};

cudaError_t rmsnorm_rows_launch(const float *x, const float *w, float eps, float *out, int dim, int n,
                                const uint8_t *active, cudaStream_t stream, void *hi, void *lo, bool programmatic) {
    RowLaunch l(n, kNormThreads, stream, programmatic);
    return cudaLaunchKernelEx(&l.cfg, rmsnorm_rows_kernel, x, w, eps, out, dim, active, static_cast<uint2 *>(hi),
                              static_cast<uint2 *>(lo));
}

cudaError_t swiglu_rows_launch(float *g, const float *u, int hidden, int n, cudaStream_t stream, void *hi, void *lo,
                               bool programmatic) {
    const size_t total4 = size_t(hidden) * n / 4;
    const int grid = static_cast<int>((total4 + 255) / 256 < 148 * 8 ? (total4 + 255) / 256 : 148 * 8);
    RowLaunch l(grid, 256, stream, programmatic);
    return cudaLaunchKernelEx(&l.cfg, swiglu_rows_kernel, reinterpret_cast<float4 *>(g), reinterpret_cast<const float4 *>(u),
                              total4, static_cast<uint2 *>(hi), static_cast<uint2 *>(lo));
}

cudaError_t kv_append_launch(const float *k, const float *v, const float *rope_cos, const float *rope_sin,
                             const int32_t *positions, const int32_t *slots, const uint8_t *active,
                             KvGeom kv, int layer, int head_dim, int n, cudaStream_t stream, bool programmatic) {
    RowLaunch l(n, 256, stream, programmatic);
    return cudaLaunchKernelEx(&l.cfg, kv_append_kernel, k, v, rope_cos, rope_sin, positions, slots, active, kv, layer, head_dim);
}

cudaError_t argmax_rows_launch(const float *logits, int vocab, int n, const uint8_t *active, int32_t *out,
                               cudaStream_t stream, bool programmatic) {
    RowLaunch l(n, 1024, stream, programmatic);
    return cudaLaunchKernelEx(&l.cfg, argmax_rows_kernel, logits, vocab, active, out);
}

cudaError_t add_rows_launch(float *x, const float *y, size_t total, cudaStream_t stream, bool programmatic) {
    const int grid = static_cast<int>((total + 1023) / 1024 < 148 * 8 ? (total + 1023) / 1024 : 148 * 8);
    RowLaunch l(grid, 256, stream, programmatic);
    return cudaLaunchKernelEx(&l.cfg, add_rows_kernel, x, y, total);
}

cudaError_t split_rows_launch(const float *x, size_t total, void *hi, void *lo, cudaStream_t stream, bool programmatic) {
    const size_t total4 = total / 4;  // row lengths are multiples of 256
    const int grid = static_cast<int>((total4 + 255) / 256 < 148 * 8 ? (total4 + 255) / 256 : 148 * 8);
    RowLaunch l(grid, 256, stream, programmatic);
    return cudaLaunchKernelEx(&l.cfg, split_rows_kernel, reinterpret_cast<const float4 *>(x), total4, static_cast<uint2 *>(hi),
                              static_cast<uint2 *>(lo));
}

cudaError_t tp_pack_best_launch(const float *logits, const int32_t *idx, int l_vocab, int index_offset, int n,
                                float *best, cudaStream_t stream) {
    tp_pack_best_kernel<<<(n + 127) / 128, 128, 0, stream>>>(logits, idx, l_vocab, index_offset, n, best);
    return cudaGetLastError();
}

cudaError_t tp_pick_best_launch(const float *all, int ranks, int n, const uint8_t *active, int32_t *out,
                                cudaStream_t stream) {
    tp_pick_best_kernel<<<(n + 127) / 128, 128, 0, stream>>>(all, ranks, n, active, out);
    return cudaGetLastError();
}

cudaError_t fill_launch(uint32_t *buf, size_t words, uint32_t value, cudaStream_t stream) {
    fill_kernel<<<148 * 8, 256, 0, stream>>>(buf, words, value);
    return cudaGetLastError();
}

}  // namespace jl
