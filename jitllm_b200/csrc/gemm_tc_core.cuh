// What the tensor-core (tcgen05) matrix-matrix kernels share: waits, tensor-memory access, the conversion of
// quantised units into binary16 operands and the cut of the work list into equal ranges.
#pragma once

#include "gemm_tc.cuh"

#include "formats.cuh"

#include <cuda.h>
#include <cuda_fp16.h>

namespace jl {
namespace {

// Which bounded wait the kernel uses (a build-time experiment switch).
#define GEMM_WAIT mbar_poll_bounded

constexpr int kTileM = 128;    // weight rows per tile
constexpr int kRawK = 256;     // columns per raw stage (one Q4_K super-block per row)

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// One box of a 2-D tensor map into shared memory; x counts 32-bit words along a row (x * 4 bytes is
// a multiple of 16 for every raw stage: 144- and 272-byte steps), y counts rows.
__device__ __forceinline__ void tma_load_2d(void *dst_smem, const CUtensorMap *map, int x, int y, uint64_t *bar,
                                            uint64_t policy) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint "
        "[%0], [%1, {%2, %3}], [%4], %5;" ::"r"(smem_u32(dst_smem)),
        "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar)), "l"(policy)
        : "memory");
}

__device__ __forceinline__ void tma_load_2d_plain(void *dst_smem, const CUtensorMap *map, int x, int y, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(smem_u32(dst_smem)), "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_u32(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// mbar_poll_bounded on a shared-window address.
__device__ __forceinline__ bool mbar_poll_bounded_u32(uint32_t bar, uint32_t parity, uint32_t limit = (1u << 24)) {
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
        __nanosleep(40);
    }
    return false;
}
// 16 consecutive 32-bit columns of this thread's lane.
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// 32 lanes x 16 consecutive fp32 columns of the accumulator into registers.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// Shared-memory matrix descriptor of the B operand: K-major, 128-byte swizzle, rows of 64 fp16
// (128 B), groups of eight rows 1024 B apart. Low word: bits 0-13 the start address in 16-byte
// units, bit 16 the (unused) leading byte offset; high word: bits 0-13 the stride between 8-row
// groups in 16-byte units (1024 >> 4), bit 14 the descriptor version for sm_100, bits 29-31 the
// swizzle mode (2 = 128 bytes). The issuing thread keeps the low word as a running value.
constexpr uint32_t kSw128DescHi = uint32_t(1024 >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint32_t sw128_desc_lo(uint32_t smem_addr) { return ((smem_addr >> 4) & 0x3FFFu) | (1u << 16); }
// 16-byte chunk c of row r inside a [rows][64 fp16] swizzled tile.
__device__ __forceinline__ uint32_t sw128_offset(int r, int c) { return uint32_t(r) * 128u + uint32_t((c ^ (r & 7)) << 4); }

__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
    const __half2 h = __halves2half2(__float2half_rn(a), __float2half_rn(b));
    return *reinterpret_cast<const uint32_t *>(&h);
}



template <int TYPE>
struct RawFmt {
    static constexpr int row_bytes = TYPE == kQ8_0   ? 272  // 256 columns of one row
                                     : TYPE == kQ6_K ? kQ6_KPadded
                                     : TYPE == kQ5_K ? kQ5_KBytes
                                     : TYPE == kQ4_1 ? 8 * kQ4_1Bytes
                                                     : 144;
    static constexpr int stage_bytes = kTileM * row_bytes;
};

// Two bytes of v (selected by sel) as half2 {1024 + byte, 1024 + byte}: 0x64xx is 1024 + xx in fp16.
__device__ __forceinline__ __half2 bytes_to_half2_plus1024(uint32_t v, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(v), "r"(0x64646464u), "r"(sel));
    return *reinterpret_cast<const __half2 *>(&r);
}
__device__ __forceinline__ uint32_t h2_bits(__half2 h) { return *reinterpret_cast<const uint32_t *>(&h); }

// Operand order. Inside every group of four consecutive K elements the tensor-memory columns (and the
// activation rows, see the in-kernel activation conversion below and split4_store in ops.cu) hold
// the pairs (k0, k2) and (k1, k3): a sum over K does not care about the order as long as both
// operands agree, and the bytes 0 and 2 of a 32-bit word come out together with one logic operation.

// What a thread keeps of its 64-weight unit between the two 32-weight halves it converts.
template <int TYPE>
struct UnitRegs;

template <>
struct UnitRegs<kQ4_K> {
    uint32_t qw[8];         // the unit's 32 bytes: low nibbles = first half, high nibbles = second
    __half2 d2;             // the super-block scale, exact (it is stored as binary16)
    __half2 sc2[2], off2[2];  // per half: the 6-bit scale as a number, and -base * scale
    __half2 chi2[2], clo2[2];  // per half: -dmin * m as an exact binary16 pair (17 significant bits)
};
template <>
struct UnitRegs<kQ4_0> {
    uint32_t t[9];  // two 18-byte blocks
};
template <>
struct UnitRegs<kQ8_0> {
    uint32_t base;  // shared address of the unit (two 34-byte blocks); its halves are loaded one at a time
};
template <>
struct UnitRegs<kQ5_K> {
    uint32_t qw[8];            // as Q4_K
    __half2 d2;
    __half2 sc2[2], off2[2];
    __half2 chi2[2], clo2[2];
    uint32_t qh_at;            // shared address of the super-block's 32 bytes of fifth bits (read again per half)
    int shift;                 // bit of those bytes that belongs to the unit's low nibbles (the high nibbles' is the next)
};
template <>
struct UnitRegs<kQ4_1> {
    uint32_t t[10];  // two 20-byte blocks: (d, m), 16 bytes of nibbles, twice
};
template <>
struct UnitRegs<kQ6_K> {
    uint32_t blk;   // shared address of the (padded) super-block; the unit's halves are loaded one at a time
    int unit;
    __half2 d2;     // the super-block scale, exact (it is stored as binary16)
};

__device__ __forceinline__ __half2 u32_as_half2(uint32_t v) { return *reinterpret_cast<const __half2 *>(&v); }

// Loads a unit: `row_u32` is the shared address of the row's 256-column slice of a raw stage, `unit`
// the 64-column unit inside it (0..3).
template <int TYPE>
__device__ __forceinline__ void unit_load(uint32_t row_u32, int unit, UnitRegs<TYPE> &r) {
    if constexpr (TYPE == kQ4_K || TYPE == kQ5_K) {
        // tensor/standard/Q4_KFloatTensor.java:68-122: unit p holds sub-blocks 2p (low nibbles) and
        // 2p+1 (high nibbles) of the same 32 bytes; w = (d*sc)*q - dmin*m. Q5_K (Q5_KFloatTensor.java:87-127) is
        // the same with 32 bytes of fifth bits between the header and the nibbles.
        constexpr int kNibbles = TYPE == kQ5_K ? 48 : 16;
        const uint4 hdr = lds128(row_u32);
        const uint4 q0 = lds128(row_u32 + kNibbles + unit * 32);
        const uint4 q1 = lds128(row_u32 + kNibbles + 16 + unit * 32);
        if constexpr (TYPE == kQ5_K) {
            r.qh_at = row_u32 + 16;
            r.shift = 2 * unit;
        }
        r.qw[0] = q0.x; r.qw[1] = q0.y; r.qw[2] = q0.z; r.qw[3] = q0.w;
        r.qw[4] = q1.x; r.qw[5] = q1.y; r.qw[6] = q1.z; r.qw[7] = q1.w;
        r.d2 = u32_as_half2(__byte_perm(hdr.x, 0u, 0x1010));
        const float dmin = half_bits_to_float(hdr.x >> 16);
        uint32_t scw, mw;
        if (unit < 2) {
            scw = hdr.y & 0x3F3F3F3Fu;
            mw = hdr.z & 0x3F3F3F3Fu;
        } else {
            scw = (hdr.w & 0x0F0F0F0Fu) | ((hdr.y >> 2) & 0x30303030u);
            mw = ((hdr.w >> 4) & 0x0F0F0F0Fu) | ((hdr.z >> 2) & 0x30303030u);
        }
        const int sh = (unit & 1) * 16;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            // 0x6400 | n is 1024 + n in binary16: the 6-bit scale and minimum become numbers without
            // the conversion unit.
            const uint32_t scb = (scw >> (sh + 8 * h)) & 0xFFu, mb = (mw >> (sh + 8 * h)) & 0xFFu;
            const __half2 k1024 = u32_as_half2(0x64006400u);
            r.sc2[h] = __hsub2(u32_as_half2(0x64006400u | scb | (scb << 16)), k1024);
            r.off2[h] = __hmul2(r.sc2[h], u32_as_half2(h == 0 ? 0xE400E400u : 0xD400D400u));  // * -1024, * -64: exact
            const float c = -__fmul_rn(dmin, __half2float(__low2half(__hsub2(u32_as_half2(0x64006400u | mb), k1024))));
            const __half chi = __float2half_rn(c);
            const __half clo = __float2half_rn(c - __half2float(chi));  // exact: c has 17 significant bits
            r.chi2[h] = __half2half2(chi);
            r.clo2[h] = __half2half2(clo);
        }
    } else if constexpr (TYPE == kQ4_0) {
        const uint32_t base = row_u32 + unit * 36;
#pragma unroll
        for (int i = 0; i < 9; ++i) r.t[i] = lds32(base + 4 * i);
    } else if constexpr (TYPE == kQ4_1) {
        const uint32_t base = row_u32 + unit * 40;
#pragma unroll
        for (int i = 0; i < 10; ++i) r.t[i] = lds32(base + 4 * i);
    } else if constexpr (TYPE == kQ6_K) {
        r.blk = row_u32;
        r.unit = unit;
        const uint32_t dw = lds32(row_u32 + 208) & 0xFFFFu;
        r.d2 = u32_as_half2(dw | (dw << 16));
    } else {
        r.base = row_u32 + unit * 68;
    }
}

// 32 of the unit's 64 consecutive weights as 16 tensor-memory columns, each weight rounded to binary16:
// `half` 0 = the first 32 weights, 1 = the next 32. The two halves are converted and stored one after
// the other so that only 16 results are live.
template <int TYPE>
__device__ __forceinline__ void unit_convert(const UnitRegs<TYPE> &r, int half, uint32_t (&out)[16]) {
    if constexpr (TYPE == kQ4_K) {
        // The conversion runs on the floating-point pipe, two weights per instruction: one logic
        // operation drops two nibbles into the mantissas of a binary16 pair (0x6400 | q = 1024 + q for
        // the low nibbles, 0x5400 | (q << 4) = 64 + q for the high ones, both exact), one fused
        // multiply-add makes t = sc * q out of it (an integer below 1024: exact), a second one
        // d * t + c_hi rounds once, and the last addition brings in c_lo, the 6 bits of dmin * m that
        // c_hi cannot hold. The result is within two binary16 roundings of d * sc * q - dmin * m.
        const uint32_t mask = half == 0 ? 0x000F000Fu : 0x00F000F0u, magic = half == 0 ? 0x64006400u : 0x54005400u;
        const __half2 sc2 = r.sc2[half], off2 = r.off2[half], chi2 = r.chi2[half], clo2 = r.clo2[half];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const __half2 e = u32_as_half2((r.qw[i] & mask) | magic);         // bytes 0 and 2 of the word
            const __half2 o = u32_as_half2(((r.qw[i] >> 8) & mask) | magic);  // bytes 1 and 3
            const __half2 we = __hadd2(__hfma2(r.d2, __hfma2(sc2, e, off2), chi2), clo2);
            const __half2 wo = __hadd2(__hfma2(r.d2, __hfma2(sc2, o, off2), chi2), clo2);
            out[2 * i] = h2_bits(we);
            out[2 * i + 1] = h2_bits(wo);
        }
    } else if constexpr (TYPE == kQ5_K) {
        // As Q4_K, with the fifth bit dropped into the same mantissa: 1024 + q (low nibbles: bit 4) or 64 + q (high
        // nibbles, whose mantissa unit is 1/16: bit 8). sc * q stays below 2048, exact in binary16.
        const uint32_t mask = half == 0 ? 0x000F000Fu : 0x00F000F0u, magic = half == 0 ? 0x64006400u : 0x54005400u;
        const __half2 sc2 = r.sc2[half], off2 = r.off2[half], chi2 = r.chi2[half], clo2 = r.clo2[half];
        const uint4 f0 = lds128(r.qh_at), f1 = lds128(r.qh_at + 16);
        const uint32_t fw[8] = {f0.x, f0.y, f0.z, f0.w, f1.x, f1.y, f1.z, f1.w};
        const int fs = r.shift + half;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t f = fw[i] >> fs;  // bit 0 of every byte: the fifth bit of that weight
            const uint32_t fe = half == 0 ? ((f << 4) & 0x00100010u) : ((f << 8) & 0x01000100u);  // bytes 0 and 2
            const uint32_t fo = half == 0 ? ((f >> 4) & 0x00100010u) : (f & 0x01000100u);          // bytes 1 and 3
            const __half2 e = u32_as_half2((r.qw[i] & mask) | fe | magic);
            const __half2 o = u32_as_half2(((r.qw[i] >> 8) & mask) | fo | magic);
            const __half2 we = __hadd2(__hfma2(r.d2, __hfma2(sc2, e, off2), chi2), clo2);
            const __half2 wo = __hadd2(__hfma2(r.d2, __hfma2(sc2, o, off2), chi2), clo2);
            out[2 * i] = h2_bits(we);
            out[2 * i + 1] = h2_bits(wo);
        }
    } else if constexpr (TYPE == kQ4_1) {
        // tensor/standard/Q4_1FloatTensor.java:76-99: a unit is two 20-byte blocks; w = q * d + m with an unsigned
        // nibble, one fused multiply-add on exact inputs.
        const uint32_t hdr = r.t[5 * half];
        const __half2 d2 = u32_as_half2(__byte_perm(hdr, 0u, 0x1010)), m2 = u32_as_half2(__byte_perm(hdr, 0u, 0x3232));
        const __half2 off = __float2half2_rn(1024.0f);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t q = r.t[5 * half + 1 + i];
            const uint32_t l4 = q & 0x0F0F0F0Fu, h4 = (q >> 4) & 0x0F0F0F0Fu;
            out[2 * i] = h2_bits(__hfma2(__hsub2(bytes_to_half2_plus1024(l4, 0x4240u), off), d2, m2));
            out[2 * i + 1] = h2_bits(__hfma2(__hsub2(bytes_to_half2_plus1024(l4, 0x4341u), off), d2, m2));
            out[8 + 2 * i] = h2_bits(__hfma2(__hsub2(bytes_to_half2_plus1024(h4, 0x4240u), off), d2, m2));
            out[8 + 2 * i + 1] = h2_bits(__hfma2(__hsub2(bytes_to_half2_plus1024(h4, 0x4341u), off), d2, m2));
        }
    } else if constexpr (TYPE == kQ6_K) {
        // tensor/standard/Q6_KFloatTensor.java:64-117. Unit p = 2h + u of the super-block: half h, the groups 2u
        // (this call's half 0) and 2u + 1 (half 1) of 32 weights: nibble u of ql[64 h + 32 half + j], bits
        // 4u + 2 half .. +1 of qh[32 h + j], one signed byte scale per 16 weights; w = d * scale * (v - 32).
        // v - 32 is exact in binary16; d * scale has up to 18 significant bits and is applied as an exact
        // binary16 pair (hi, lo): w = (v - 32) * hi + (v - 32) * lo, one rounding apart from the small lo product.
        const int h = r.unit >> 1, u = r.unit & 1;
        const uint32_t ql_at = r.blk + 64 * h + 32 * half, qh_at = r.blk + 128 + 32 * h;
        const uint32_t scw = lds32(r.blk + 192 + 8 * h + 4 * u) >> (16 * half);  // bytes 0, 1: this half's two scales
        const float d = __half2float(__low2half(r.d2));
        __half2 hi2[2], lo2[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const float ds = __fmul_rn(d, static_cast<float>(static_cast<int>(static_cast<int8_t>((scw >> (8 * k)) & 0xFFu))));
            const __half hi = __float2half_rn(ds);
            hi2[k] = __half2half2(hi);
            lo2[k] = __half2half2(__float2half_rn(ds - __half2float(hi)));
        }
        const __half2 off = __float2half2_rn(1056.0f);  // 1024 of the byte trick + 32
        const int qsh = 4 * u + 2 * half;
#pragma unroll
        for (int q = 0; q < 2; ++q) {  // four words at a time: one 16-byte load of each plane, one scale
            const uint4 l4 = lds128(ql_at + 16 * q), h4 = lds128(qh_at + 16 * q);
            const uint32_t lw[4] = {l4.x, l4.y, l4.z, l4.w}, hw[4] = {h4.x, h4.y, h4.z, h4.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t v = ((lw[i] >> (4 * u)) & 0x0F0F0F0Fu) | (((hw[i] >> qsh) << 4) & 0x30303030u);
                const __half2 e = __hsub2(bytes_to_half2_plus1024(v, 0x4240u), off);
                const __half2 o = __hsub2(bytes_to_half2_plus1024(v, 0x4341u), off);
                out[8 * q + 2 * i] = h2_bits(__hfma2(e, hi2[q], __hmul2(e, lo2[q])));
                out[8 * q + 2 * i + 1] = h2_bits(__hfma2(o, hi2[q], __hmul2(o, lo2[q])));
            }
        }
    } else if constexpr (TYPE == kQ4_0) {
        // tensor/standard/Q4_0FloatTensor.java:56-79: a unit is two 18-byte blocks; element i < 16
        // is the low nibble of byte i, element i >= 16 the high nibble of byte i - 16; w = (q-8)*d.
        // (q-8) is exact in fp16 and d is fp16, so one half-precision multiply rounds exactly like
        // the reference's fp32 product narrowed to fp16.
        const uint32_t dbits = half == 0 ? (r.t[0] & 0xFFFFu) : (r.t[4] >> 16);
        const __half2 d2 = u32_as_half2(dbits | (dbits << 16));
        const __half2 off = __float2half2_rn(1032.0f);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t q = half == 0 ? __funnelshift_r(r.t[i], r.t[i + 1], 16) : r.t[5 + i];
            const uint32_t l4 = q & 0x0F0F0F0Fu, h4 = (q >> 4) & 0x0F0F0F0Fu;
            out[2 * i] = h2_bits(__hmul2(__hsub2(bytes_to_half2_plus1024(l4, 0x4240u), off), d2));
            out[2 * i + 1] = h2_bits(__hmul2(__hsub2(bytes_to_half2_plus1024(l4, 0x4341u), off), d2));
            out[8 + 2 * i] = h2_bits(__hmul2(__hsub2(bytes_to_half2_plus1024(h4, 0x4240u), off), d2));
            out[8 + 2 * i + 1] = h2_bits(__hmul2(__hsub2(bytes_to_half2_plus1024(h4, 0x4341u), off), d2));
        }
    } else {
        // tensor/standard/Q8_0FloatTensor.java:53-61: a unit is two 34-byte blocks; w = q * d, again
        // one exact-input half-precision multiply.
        const uint32_t base = r.base + half * 32;
        uint32_t t[9];
#pragma unroll
        for (int i = 0; i < 9; ++i) t[i] = lds32(base + 4 * i);
        const uint32_t dbits = half == 0 ? (t[0] & 0xFFFFu) : (t[0] >> 16);
        const __half2 d2 = u32_as_half2(dbits | (dbits << 16));
        const __half2 off = __float2half2_rn(1152.0f);  // 1024 + the 128 added by the sign flip
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t q = (half == 0 ? __funnelshift_r(t[i], t[i + 1], 16) : t[1 + i]) ^ 0x80808080u;
            out[2 * i] = h2_bits(__hmul2(__hsub2(bytes_to_half2_plus1024(q, 0x4240u), off), d2));
            out[2 * i + 1] = h2_bits(__hmul2(__hsub2(bytes_to_half2_plus1024(q, 0x4341u), off), d2));
        }
    }
}

struct TileRef {
    int seg, row0;
};

__device__ __forceinline__ TileRef locate_tile(const GemmArgs &a, int tile) {
    TileRef t = {0, 0};
    for (int s = 0; s < a.nseg; ++s) {
        const int tiles = (a.seg[s].rows + kTileM - 1) / kTileM;
        if (tile < tiles || s == a.nseg - 1) {
            t.seg = s;
            t.row0 = tile * kTileM;
            return t;
        }
        tile -= tiles;
    }
    return t;
}

// The contiguous range of the flattened work list that CTA c owns.
// (The launcher refuses work lists with total * ctas >= 2^32, so the arithmetic stays in 32 bits: a
// 64-bit division costs about a hundred instructions, and these run at every tile end.)
__device__ __forceinline__ int range_lo(int total, int c, int ctas) {
    return int(uint32_t(total) * uint32_t(c) / uint32_t(ctas));
}
__device__ __forceinline__ int cta_of(int total, int f, int ctas) {
    int c = int(uint32_t(f) * uint32_t(ctas) / uint32_t(total));
    while (c + 1 < ctas && range_lo(total, c + 1, ctas) <= f) ++c;
    while (c > 0 && range_lo(total, c, ctas) > f) --c;
    return c;
}

}  // namespace
}  // namespace jl
