// What the decode matvec kernels (okf_gemv.cu, okf_gemv_stream.cu) work on: the integer MMA, a unit's arithmetic for one column,
// and how x becomes bytes in shared memory.  (Several columns: okf_gemv_wide.cuh.)
#pragma once
#include "okf_gemv_mma.cuh"
#include "okf_gemv_wide.cuh"

namespace okf {

template <int TY> struct UnitGeom;
template <> struct UnitGeom<T_Q4_K> { static constexpr uint32_t bytes = 144; };
template <> struct UnitGeom<T_Q8_0> { static constexpr uint32_t bytes = 272; };
template <> struct UnitGeom<T_Q4_0> { static constexpr uint32_t bytes = 144; };
template <> struct UnitGeom<T_Q6_K> { static constexpr uint32_t bytes = 210; };
template <> struct UnitGeom<T_Q5_K> { static constexpr uint32_t bytes = 176; };
template <> struct UnitGeom<T_IQ4_NL> { static constexpr uint32_t bytes = 144; };
template <> struct UnitGeom<T_Q2_0> { static constexpr uint32_t bytes = 68; };
template <> struct UnitGeom<T_IQ2_XXS> { static constexpr uint32_t bytes = 66; };

constexpr uint32_t kZeroOff = 256;    // what the lanes that feed nothing into an MMA read instead of x
constexpr uint32_t kConsumers = kGemvWarps * 32;
// WIDE x panel: a unit of a byte column is its 256 bytes in k order, except that in
// quarters 2 and 3 neighbouring 16-byte pieces are swapped; with the second byte column
// 32 (mod 128) bytes after the first, the lanes of a load that carry data touch different
// bank groups.
constexpr uint32_t kXqUnit = 256;
constexpr float kXqMax = 32512.f;  // 127 * 256: hi stays a signed byte after rounding
// SEP x panel: per byte column and unit, four quarters of 80 bytes: 64 bytes of x in k
// order (two types: see stage_x_bytes), then in the first byte column the quarter's record {scale,
// scale * sum of x over its first 32-wide block, over its second, -}, in the second one, for Q6_K,
// the sums over its 16-wide groups.  One address register reaches a
// quarter's x and its record with immediate offsets.  80-byte quarters put the four
// quarters of a 16-byte access on different bank groups (0, 80, 32, 112 mod 128) and the
// second byte column, 64 (mod 128) bytes after the first, on the other four.
constexpr uint32_t kSepQuarter = 80, kSepUnit = 4 * kSepQuarter;

__host__ __device__ inline uint32_t xq_col_stride(uint32_t units) {
    const uint32_t raw = units * kXqUnit;
    return raw + ((32u + 128u - raw % 128u) % 128u);
}
__host__ __device__ inline uint32_t sep_col_stride(uint32_t units) {
    const uint32_t raw = units * kSepUnit;
    return raw + ((64u + 128u - raw % 128u) % 128u);
}
__host__ __device__ inline uint32_t xq_piece_offset(uint32_t c, uint32_t piece) {
    return c * 64 + ((piece ^ (c >> 1)) & 3u) * 16;
}

// ---- integer MMA: D (16 x 8, s32) += A (16 x 32, bytes) * B (32 x 8, signed bytes) ----
// Thread (g = lane / 4, c = lane % 4): a0 / a2 = row g, a1 / a3 = row g + 8, at
// k-slots 4c..4c+3 (a0, a1, b0) and 16+4c..16+4c+3 (a2, a3, b1); b = column g;
// d[0], d[1] = row g, columns 2c, 2c+1; d[2], d[3] = row g + 8.
template <bool SIGNED_A>
__device__ __forceinline__ void imma(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                     uint32_t b1) {
    if constexpr (SIGNED_A)
        asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    else
        asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// first of a chain: D = A * B
template <bool SIGNED_A>
__device__ __forceinline__ void imma0(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                      uint32_t b1) {
    if constexpr (SIGNED_A)
        asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
            : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
    else
        asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
            : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}
// sum over the hi and lo bytes of x: columns 2c (hi) and 2c+1 (lo) of one row
__device__ __forceinline__ float join_hi_lo(int hi, int lo) { return (float)(hi * 256 + lo); }

// ---- per-unit arithmetic, SEP -------------------------------------------------
// What a thread works out once per launch for the one-column path.
struct SepConst {
    uint32_t qoff;          // where this thread's share of a unit starts (bytes from the unit's start)
    uint32_t hoff;          // Q2_0: where the block that share lies in starts
    uint32_t sel, m1, m2;   // Q4_K: how to pick this thread's 6-bit scales and mins out of the 12 bytes
    bool low;               // Q4_K: sub-blocks 0..3 (plain 6-bit fields) or 4..7 (split fields)
};
template <int TY>
__device__ __forceinline__ SepConst sep_const(uint32_t c) {
    SepConst k = {};
    if constexpr (TY == T_Q4_K || TY == T_Q5_K) {
        k.qoff = (TY == T_Q4_K ? 16 : 48) + 32 * c;
        k.hoff = 2 * c;  // Q5_K: the bit of qh that belongs to sub-block 2c; the next one is sub-block 2c + 1's
        k.sel = (c & 1) ? 0x7632u : 0x5410u;
        k.low = c < 2;
        k.m1 = k.low ? 0x3F3F3F3Fu : 0x0F0F0F0Fu;
        k.m2 = k.low ? 0u : 0x30303030u;
    } else if constexpr (TY == T_Q8_0) {
        k.qoff = 68 * c;
    } else if constexpr (TY == T_Q4_0 || TY == T_IQ4_NL) {
        k.qoff = 36 * c;
    } else if constexpr (TY == T_Q6_K) {
        k.qoff = 64 * (c >> 1) + 32 * (c & 1);      // 32 bytes of ql
        k.hoff = 128 + 32 * (c >> 1);               // the half's 32 bytes of qh
        k.sel = 192 + 8 * (c >> 1) + 2 * (c & 1);   // two scales, and two more 4 bytes on
        k.m1 = 0x03030303u << (2 * (c & 1));        // this thread's two bits of qh for the low nibbles
        k.m2 = 16u >> (2 * (c & 1));                // what puts those bits above a nibble
    } else if constexpr (TY == T_Q2_0) {
        k.hoff = 34 * (c >> 1);
        k.qoff = k.hoff + 2 + 16 * (c & 1);
    } else {
        k.qoff = 2 + 16 * c;
    }
    return k;
}

// ua / ub: shared addresses of the unit in rows g and g + 8.  xf: this thread's 64
// bytes of x (its quarter of the unit, the byte column its MMA column stands for; zeros
// in the lanes that feed nothing).  xi: {scale of x in this unit, scale * sum of x over
// the first 32-wide block of the quarter, over the second, -} as float bits.
// acc: rows g and g + 8.
template <int TY>
__device__ __forceinline__ void unit_sep(uint32_t ua, uint32_t ub, const SepConst &K, const Iq2Tab &tab, const uint32_t (&xf)[16],
                                         const uint4 &xi, const uint4 &xj, float (&acc)[2]) {
    const float xs = __uint_as_float(xi.x);
    if constexpr (TY == T_Q4_K) {
        // {f16 d; f16 dmin; u8 scales[12]; u8 qs[128]} (LLM/Quantize/KQuants.swift:104-125).
        // Group c of qs (32 bytes): low nibbles = sub-block 2c, high = 2c+1, both in k order.
        // The high nibbles stay where they are (16 x the value); the sums are shifted back.
        const uint4 ha = lds128(ua), hb = lds128(ub);
        const uint4 a0 = lds128(ua + K.qoff), a1 = lds128(ua + K.qoff + 16);
        const uint4 b0 = lds128(ub + K.qoff), b1 = lds128(ub + K.qoff + 16);
        const uint32_t wa[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
        const uint32_t wb[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
        const uint32_t ml = 0x0F0F0F0Fu, mh = 0xF0F0F0F0u;
        int lo[4], hi[4];
        imma0<false>(lo, wa[0] & ml, wb[0] & ml, wa[1] & ml, wb[1] & ml, xf[0], xf[1]);
        imma0<false>(hi, wa[0] & mh, wb[0] & mh, wa[1] & mh, wb[1] & mh, xf[8], xf[9]);
#pragma unroll
        for (int i = 1; i < 4; i++) {
            imma<false>(lo, wa[2 * i] & ml, wb[2 * i] & ml, wa[2 * i + 1] & ml, wb[2 * i + 1] & ml, xf[2 * i], xf[2 * i + 1]);
            imma<false>(hi, wa[2 * i] & mh, wb[2 * i] & mh, wa[2 * i + 1] & mh, wb[2 * i + 1] & mh, xf[8 + 2 * i],
                        xf[9 + 2 * i]);
        }
        // 6-bit (scale, min) of sub-blocks 2c and 2c+1 of both rows (ggml get_scale_min_k4,
        // LLM/Quantize/KQuants.swift:86-101) as bytes {row a: 2c, 2c+1, row b: 2c, 2c+1},
        // without a branch: the two cases differ in where the low bits come from.
        const uint32_t pa = prmt(ha.y, hb.y, K.sel), pb = prmt(ha.z, hb.z, K.sel), pe = prmt(ha.w, hb.w, K.sel);
        const uint32_t sc = ((K.low ? pa : pe) & K.m1) | ((pa >> 2) & K.m2);
        const uint32_t mn = ((K.low ? pb : (pe >> 4)) & K.m1) | ((pb >> 2) & K.m2);
        // From here on floating point: integer instructions run at half the rate of fp32 ones
        // on this part, and the masks above have used up the integer budget.  A scale byte
        // becomes a float with one byte permute and one subtraction.  The high-nibble sums
        // carry a factor 16 that goes into x's scale.
        const float xs16 = xs * 0.0625f;
        const float la = join_hi_lo(lo[0], lo[1]), ha_ = join_hi_lo(hi[0], hi[1]);
        const float lb = join_hi_lo(lo[2], lo[3]), hb_ = join_hi_lo(hi[2], hi[3]);
        const float x0 = __uint_as_float(xi.y), x1 = __uint_as_float(xi.z);  // scale * sum of x per block
        const float2 fa = __half22float2(*reinterpret_cast<const __half2 *>(&ha.x));
        const float2 fb = __half22float2(*reinterpret_cast<const __half2 *>(&hb.x));
        acc[0] += fa.x * (byte_to_f32(sc, 0) * (xs * la) + byte_to_f32(sc, 1) * (xs16 * ha_)) -
                  fa.y * (byte_to_f32(mn, 0) * x0 + byte_to_f32(mn, 1) * x1);
        acc[1] += fb.x * (byte_to_f32(sc, 2) * (xs * lb) + byte_to_f32(sc, 3) * (xs16 * hb_)) -
                  fb.y * (byte_to_f32(mn, 2) * x0 + byte_to_f32(mn, 3) * x1);
    } else if constexpr (TY == T_Q4_0) {
        // eight blocks {f16 d; u8 qs[16]}, byte j = weights j (low nibble) and j + 16 (high), value
        // (q - 8) * d (LLM/Gemma/Gemma4Quant.swift:30-49).  Thread c takes blocks 2c and 2c+1:
        // {d0, qs0[16], d1, qs1[16]} = 9 words (units start on 16-byte boundaries, 36c is a
        // multiple of 4).  Nibbles are masked in place; the high ones stay 16 x the value.
        uint32_t wa[9], wb[9];
#pragma unroll
        for (int i = 0; i < 9; i++) {
            wa[i] = lds32(ua + K.qoff + 4 * i);
            wb[i] = lds32(ub + K.qoff + 4 * i);
        }
        uint32_t qa[8], qb[8];  // block 0's bytes start two bytes into word 0, block 1's on word 5
#pragma unroll
        for (int i = 0; i < 4; i++) {
            qa[i] = __funnelshift_r(wa[i], wa[i + 1], 16);
            qb[i] = __funnelshift_r(wb[i], wb[i + 1], 16);
            qa[4 + i] = wa[5 + i];
            qb[4 + i] = wb[5 + i];
        }
        const uint32_t ml = 0x0F0F0F0Fu, mh = 0xF0F0F0F0u;
        float part[2][2];  // [block][row]: sum of q * x in units of x's scale
#pragma unroll
        for (int blk = 0; blk < 2; blk++) {
            const uint32_t *a = qa + 4 * blk, *b = qb + 4 * blk;
            const uint32_t *xb = xf + 8 * blk;  // bytes of k 0..15 (low nibbles), then 16..31 (high)
            int lo[4], hi[4];
            imma0<false>(lo, a[0] & ml, b[0] & ml, a[1] & ml, b[1] & ml, xb[0], xb[1]);
            imma0<false>(hi, a[0] & mh, b[0] & mh, a[1] & mh, b[1] & mh, xb[4], xb[5]);
            imma<false>(lo, a[2] & ml, b[2] & ml, a[3] & ml, b[3] & ml, xb[2], xb[3]);
            imma<false>(hi, a[2] & mh, b[2] & mh, a[3] & mh, b[3] & mh, xb[6], xb[7]);
            part[blk][0] = fmaf(join_hi_lo(hi[0], hi[1]), 0.0625f, join_hi_lo(lo[0], lo[1]));
            part[blk][1] = fmaf(join_hi_lo(hi[2], hi[3]), 0.0625f, join_hi_lo(lo[2], lo[3]));
        }
        const float x0 = __uint_as_float(xi.y), x1 = __uint_as_float(xi.z);  // scale * sum of x per block
        const float da0 = f16bits(wa[0] & 0xFFFF), da1 = f16bits(wa[4] >> 16);
        const float db0 = f16bits(wb[0] & 0xFFFF), db1 = f16bits(wb[4] >> 16);
        acc[0] += da0 * fmaf(xs, part[0][0], -8.f * x0) + da1 * fmaf(xs, part[1][0], -8.f * x1);
        acc[1] += db0 * fmaf(xs, part[0][1], -8.f * x0) + db1 * fmaf(xs, part[1][1], -8.f * x1);
    } else if constexpr (TY == T_IQ4_NL) {
        // Q4_0's layout with a codebook: weight = kvalues[nibble] * d (LLM/Gemma/Gemma4Quant.swift:5-29), looked
        // up eight nibbles at a time (see iq4nl_word; x is staged in the order they come in).  (Four at a
        // time, with selectors packed first: 5120 -> 65536 73 us at 2.6 TB/s.)
        uint32_t wa[9], wb[9];
#pragma unroll
        for (int i = 0; i < 9; i++) {
            wa[i] = lds32(ua + K.qoff + 4 * i);
            wb[i] = lds32(ub + K.qoff + 4 * i);
        }
        uint32_t qa[8], qb[8];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            qa[i] = __funnelshift_r(wa[i], wa[i + 1], 16);
            qb[i] = __funnelshift_r(wb[i], wb[i + 1], 16);
            qa[4 + i] = wa[5 + i];
            qb[4 + i] = wb[5 + i];
        }
        float part[2][2];
#pragma unroll
        for (int blk = 0; blk < 2; blk++) {
            const uint32_t *a = qa + 4 * blk, *b = qb + 4 * blk;
            const uint32_t *xb = xf + 8 * blk;
            int d[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint2 va = iq4nl_word(a[i]), vb = iq4nl_word(b[i]);
                if (i == 0) imma0<true>(d, va.x, vb.x, va.y, vb.y, xb[0], xb[1]);
                else imma<true>(d, va.x, vb.x, va.y, vb.y, xb[2 * i], xb[2 * i + 1]);
            }
            part[blk][0] = join_hi_lo(d[0], d[1]);
            part[blk][1] = join_hi_lo(d[2], d[3]);
        }
        const float da0 = f16bits(wa[0] & 0xFFFF), da1 = f16bits(wa[4] >> 16);
        const float db0 = f16bits(wb[0] & 0xFFFF), db1 = f16bits(wb[4] >> 16);
        acc[0] += xs * (da0 * part[0][0] + da1 * part[1][0]);
        acc[1] += xs * (db0 * part[0][1] + db1 * part[1][1]);
    } else if constexpr (TY == T_Q5_K) {
        // {f16 d; f16 dmin; u8 scales[12]; u8 qh[32]; u8 qs[128]} (LLM/Quantize/KQuants.swift:127-158):
        // Q4_K's header and nibbles, plus a fifth bit: bit j of qh[l] for sub-block j.  As in Q6_K,
        // nibbles and bits go in where they stand and their sums are put together as integers.  (Joined into
        // bytes before the MMA: 5120 -> 65536 50 us at 4.6 TB/s.)
        const uint4 ha = lds128(ua), hb = lds128(ub);
        const uint32_t bit_lo = 0x01010101u << K.hoff, bit_hi = 0x02020202u << K.hoff;
        int lo[4], hi[4], el[4], eh[4];
#pragma unroll
        for (int half = 0; half < 2; half++) {  // 16 bytes of qs and of qh at a time
            const uint4 a = lds128(ua + K.qoff + 16 * half), b = lds128(ub + K.qoff + 16 * half);
            const uint4 ga = lds128(ua + 16 + 16 * half), gb = lds128(ub + 16 + 16 * half);
            const uint32_t *x0 = xf + 4 * half, *x1 = xf + 8 + 4 * half;
            if (half == 0) {
                imma0<false>(lo, a.x & 0x0F0F0F0Fu, b.x & 0x0F0F0F0Fu, a.y & 0x0F0F0F0Fu, b.y & 0x0F0F0F0Fu, x0[0], x0[1]);
                imma0<false>(el, ga.x & bit_lo, gb.x & bit_lo, ga.y & bit_lo, gb.y & bit_lo, x0[0], x0[1]);
                imma0<false>(hi, a.x & 0xF0F0F0F0u, b.x & 0xF0F0F0F0u, a.y & 0xF0F0F0F0u, b.y & 0xF0F0F0F0u, x1[0], x1[1]);
                imma0<false>(eh, ga.x & bit_hi, gb.x & bit_hi, ga.y & bit_hi, gb.y & bit_hi, x1[0], x1[1]);
            } else {
                imma<false>(lo, a.x & 0x0F0F0F0Fu, b.x & 0x0F0F0F0Fu, a.y & 0x0F0F0F0Fu, b.y & 0x0F0F0F0Fu, x0[0], x0[1]);
                imma<false>(el, ga.x & bit_lo, gb.x & bit_lo, ga.y & bit_lo, gb.y & bit_lo, x0[0], x0[1]);
                imma<false>(hi, a.x & 0xF0F0F0F0u, b.x & 0xF0F0F0F0u, a.y & 0xF0F0F0F0u, b.y & 0xF0F0F0F0u, x1[0], x1[1]);
                imma<false>(eh, ga.x & bit_hi, gb.x & bit_hi, ga.y & bit_hi, gb.y & bit_hi, x1[0], x1[1]);
            }
            imma<false>(lo, a.z & 0x0F0F0F0Fu, b.z & 0x0F0F0F0Fu, a.w & 0x0F0F0F0Fu, b.w & 0x0F0F0F0Fu, x0[2], x0[3]);
            imma<false>(el, ga.z & bit_lo, gb.z & bit_lo, ga.w & bit_lo, gb.w & bit_lo, x0[2], x0[3]);
            imma<false>(hi, a.z & 0xF0F0F0F0u, b.z & 0xF0F0F0F0u, a.w & 0xF0F0F0F0u, b.w & 0xF0F0F0F0u, x1[2], x1[3]);
            imma<false>(eh, ga.z & bit_hi, gb.z & bit_hi, ga.w & bit_hi, gb.w & bit_hi, x1[2], x1[3]);
        }
        // every shift is exact: the sums are multiples of what the bits stand at (and below 32 * 240 * 32512)
        auto put_lo = [&](int i) { return (float)((lo[i] * 256 + lo[i + 1]) + ((el[i] * 256 + el[i + 1]) >> K.hoff) * 16); };
        auto put_hi = [&](int i) { return (float)(((hi[i] * 256 + hi[i + 1]) >> 4) + ((eh[i] * 256 + eh[i + 1]) >> (K.hoff + 1)) * 16); };
        const uint32_t pa = prmt(ha.y, hb.y, K.sel), pb = prmt(ha.z, hb.z, K.sel), pe = prmt(ha.w, hb.w, K.sel);
        const uint32_t sc = ((K.low ? pa : pe) & K.m1) | ((pa >> 2) & K.m2);
        const uint32_t mn = ((K.low ? pb : (pe >> 4)) & K.m1) | ((pb >> 2) & K.m2);
        const float la_ = put_lo(0), ha_ = put_hi(0), lb_ = put_lo(2), hb_ = put_hi(2);
        const float x0 = __uint_as_float(xi.y), x1 = __uint_as_float(xi.z);  // scale * sum of x per block
        const float2 fa2 = __half22float2(*reinterpret_cast<const __half2 *>(&ha.x));
        const float2 fb2 = __half22float2(*reinterpret_cast<const __half2 *>(&hb.x));
        acc[0] += fa2.x * xs * (byte_to_f32(sc, 0) * la_ + byte_to_f32(sc, 1) * ha_) -
                  fa2.y * (byte_to_f32(mn, 0) * x0 + byte_to_f32(mn, 1) * x1);
        acc[1] += fb2.x * xs * (byte_to_f32(sc, 2) * lb_ + byte_to_f32(sc, 3) * hb_) -
                  fb2.y * (byte_to_f32(mn, 2) * x0 + byte_to_f32(mn, 3) * x1);
    } else if constexpr (TY == T_Q6_K) {
        // {u8 ql[128]; u8 qh[64]; i8 scales[16]; f16 d} (LLM/Quantize/KQuants.swift:160-177): weight =
        // d * scale[group of 16] * (q - 32), q = four bits of ql and two of qh.  Thread c takes 32 bytes
        // of ql, both nibbles (elements 128h + 32s + l and 64 further on; h = c / 2, s = c & 1), and
        // the two bits of the half's qh for each; x is staged to match.  Nothing is shifted or
        // joined: nibbles and bits go in where they stand, as unsigned bytes with sums of their own
        // per 16-wide scale group, which are put together as integers; 32 x the sum of x over the group leaves
        // again.  (2560 -> 151936: 86 us as signed bytes made in place, 70 us unsigned but joined
        // before the MMA and each ql byte read for one nibble.)  Units are only 2-byte aligned.
        const uint32_t sa[2] = {lds16(ua + K.sel), lds16(ua + K.sel + 4)}, sb[2] = {lds16(ub + K.sel), lds16(ub + K.sel + 4)};
        const float da = f16bits(lds16(ua + 208)), db = f16bits(lds16(ub + 208));
        uint32_t qa[8], qb[8], ha[8], hb[8];
        lds_a2<8>(ua + K.qoff, qa);
        lds_a2<8>(ub + K.qoff, qb);
        lds_a2<8>(ua + K.hoff, ha);
        lds_a2<8>(ub + K.hoff, hb);
        const uint32_t bits_lo = K.m1, bits_hi = K.m1 << 4;
        const int f = (int)K.m2;
        const float xg[4] = {__uint_as_float(xj.x), __uint_as_float(xj.y), __uint_as_float(xj.z), __uint_as_float(xj.w)};
        const float xs16 = xs * 0.0625f;
        float suma = 0.f, sumb = 0.f;
#pragma unroll
        for (int grp = 0; grp < 2; grp++) {  // 16 bytes: the low nibbles' scale group `grp`, the high nibbles' 2 + grp
            int dl[4], dh[4], el[4], eh[4];
            const uint32_t *a = qa + 4 * grp, *b = qb + 4 * grp, *va = ha + 4 * grp, *vb = hb + 4 * grp;
            const uint32_t *x0 = xf + 4 * grp, *x1 = xf + 8 + 4 * grp;
            imma0<false>(dl, a[0] & 0x0F0F0F0Fu, b[0] & 0x0F0F0F0Fu, a[1] & 0x0F0F0F0Fu, b[1] & 0x0F0F0F0Fu, x0[0], x0[1]);
            imma0<false>(el, va[0] & bits_lo, vb[0] & bits_lo, va[1] & bits_lo, vb[1] & bits_lo, x0[0], x0[1]);
            imma0<false>(dh, a[0] & 0xF0F0F0F0u, b[0] & 0xF0F0F0F0u, a[1] & 0xF0F0F0F0u, b[1] & 0xF0F0F0F0u, x1[0], x1[1]);
            imma0<false>(eh, va[0] & bits_hi, vb[0] & bits_hi, va[1] & bits_hi, vb[1] & bits_hi, x1[0], x1[1]);
            imma<false>(dl, a[2] & 0x0F0F0F0Fu, b[2] & 0x0F0F0F0Fu, a[3] & 0x0F0F0F0Fu, b[3] & 0x0F0F0F0Fu, x0[2], x0[3]);
            imma<false>(el, va[2] & bits_lo, vb[2] & bits_lo, va[3] & bits_lo, vb[3] & bits_lo, x0[2], x0[3]);
            imma<false>(dh, a[2] & 0xF0F0F0F0u, b[2] & 0xF0F0F0F0u, a[3] & 0xF0F0F0F0u, b[3] & 0xF0F0F0F0u, x1[2], x1[3]);
            imma<false>(eh, va[2] & bits_hi, vb[2] & bits_hi, va[3] & bits_hi, vb[3] & bits_hi, x1[2], x1[3]);
            // at most 16 * 16 * 63 * 32512 in magnitude (the high ones are 16 times their value): inside 32 bits
            auto put = [&](int i) { return (dl[i] + f * el[i]) * 256 + (dl[i + 1] + f * el[i + 1]); };
            auto put16 = [&](int i) { return (dh[i] + f * eh[i]) * 256 + (dh[i + 1] + f * eh[i + 1]); };
            auto scale = [&](uint32_t w) { return (float)(signed char)(grp ? w >> 8 : w & 0xFF); };
            suma = fmaf(scale(sa[0]), fmaf(xs, (float)put(0), -32.f * xg[grp]), suma);
            suma = fmaf(scale(sa[1]), fmaf(xs16, (float)put16(0), -32.f * xg[2 + grp]), suma);
            sumb = fmaf(scale(sb[0]), fmaf(xs, (float)put(2), -32.f * xg[grp]), sumb);
            sumb = fmaf(scale(sb[1]), fmaf(xs16, (float)put16(2), -32.f * xg[2 + grp]), sumb);
        }
        acc[0] = fmaf(da, suma, acc[0]);
        acc[1] = fmaf(db, sumb, acc[1]);
    } else if constexpr (TY == T_Q8_0) {
        // eight blocks {f16 d; i8 q[32]} (LLM/Gemma/Gemma4Quant.swift:51-69); thread c
        // takes blocks 2c and 2c+1: {d0, q0[32], d1, q1[32]} = 17 words (units start on
        // 16-byte boundaries, 68c is a multiple of 4); the quants go into the MMA as they are.
        uint32_t wa[17], wb[17];
#pragma unroll
        for (int i = 0; i < 17; i++) {
            wa[i] = lds32(ua + K.qoff + 4 * i);
            wb[i] = lds32(ub + K.qoff + 4 * i);
        }
        // word 0 = d0 | q0[0..1] << 16 ...: shift the first run of quants by two bytes;
        // the second run (after d1 in the high half of word 8) starts on word 9
        uint32_t qa[16], qb[16];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            qa[i] = __funnelshift_r(wa[i], wa[i + 1], 16);
            qb[i] = __funnelshift_r(wb[i], wb[i + 1], 16);
            qa[8 + i] = wa[9 + i];
            qb[8 + i] = wb[9 + i];
        }
        int lo[4], hi[4];
        imma0<true>(lo, qa[0], qb[0], qa[1], qb[1], xf[0], xf[1]);
        imma0<true>(hi, qa[8], qb[8], qa[9], qb[9], xf[8], xf[9]);
#pragma unroll
        for (int i = 1; i < 4; i++) {
            imma<true>(lo, qa[2 * i], qb[2 * i], qa[2 * i + 1], qb[2 * i + 1], xf[2 * i], xf[2 * i + 1]);
            imma<true>(hi, qa[8 + 2 * i], qb[8 + 2 * i], qa[9 + 2 * i], qb[9 + 2 * i], xf[8 + 2 * i], xf[9 + 2 * i]);
        }
        const float da0 = f16bits(wa[0] & 0xFFFF), da1 = f16bits(wa[8] >> 16);
        const float db0 = f16bits(wb[0] & 0xFFFF), db1 = f16bits(wb[8] >> 16);
        acc[0] += xs * (da0 * join_hi_lo(lo[0], lo[1]) + da1 * join_hi_lo(hi[0], hi[1]));
        acc[1] += xs * (db0 * join_hi_lo(lo[2], lo[3]) + db1 * join_hi_lo(hi[2], hi[3]));
    } else if constexpr (TY == T_Q2_0) {
        // two blocks {f16 d; u8 qs[32]} of 128 ternary codes, weight = (code - 1) * d
        // (LLM/Base/Quant.swift:2-25).  Thread c takes half (c & 1) of block c >> 1:
        // 16 bytes = 64 codes; byte t holds k 4t .. 4t+3.  Masking code s of every
        // byte of a word in place gives 4^s times the codes of k = s, 4+s, 8+s, 12+s
        // (x is staged in that order); the factors are undone on the integer sums.
        uint32_t wa[4], wb[4];
        lds_a2<4>(ua + K.qoff, wa);
        lds_a2<4>(ub + K.qoff, wb);
        const float da = f16bits(lds16(ua + K.hoff)), db = f16bits(lds16(ub + K.hoff));
        int d[4][4];  // per code position, both 32-wide halves; position s carries a factor 4^s
#pragma unroll
        for (int s = 0; s < 4; s++) {
            const uint32_t m = 0x03030303u << (2 * s);
            imma0<false>(d[s], wa[0] & m, wb[0] & m, wa[1] & m, wb[1] & m, xf[s], xf[4 + s]);
        }
#pragma unroll
        for (int s = 0; s < 4; s++) {
            const uint32_t m = 0x03030303u << (2 * s);
            imma<false>(d[s], wa[2] & m, wb[2] & m, wa[3] & m, wb[3] & m, xf[8 + s], xf[12 + s]);
        }
        int t[4];  // times 64
#pragma unroll
        for (int e = 0; e < 4; e++) t[e] = ((d[0][e] * 4 + d[1][e]) * 4 + d[2][e]) * 4 + d[3][e];
        const float xsum = __uint_as_float(xi.y) + __uint_as_float(xi.z);  // scale * sum of x over the quarter
        acc[0] += da * (xs * 0.015625f * join_hi_lo(t[0], t[1]) - xsum);
        acc[1] += db * (xs * 0.015625f * join_hi_lo(t[2], t[3]) - xsum);
    } else {
        // IQ2_XXS {f16 d; 8 x (u32 a0: four codebook indices, u32 a1: four 7-bit sign
        // indices + 4-bit scale)} (LLM/Quantize/IQ2XXS.swift:34-53).  Thread c takes
        // sub-blocks 2c and 2c+1.  A codebook entry is eight signed bytes = the two A registers
        // of a row.  (Index bytes by loads of their own, as with several columns: 17408 -> 5120 17.0 -> 19.6 us; a thread needs all four of a word.)
        uint32_t wa[4], wb[4];
        lds_a2<4>(ua + K.qoff, wa);
        lds_a2<4>(ub + K.qoff, wb);
        const float da = f16bits(lds16(ua)), db = f16bits(lds16(ub));
        float sum[2][2];
#pragma unroll
        for (int sb = 0; sb < 2; sb++) {
            const uint32_t a0a = wa[2 * sb], a1a = wa[2 * sb + 1], a0b = wb[2 * sb], a1b = wb[2 * sb + 1];
            int d[4];
#pragma unroll
            for (int l = 0; l < 4; l++) {
                const uint2 ea = tab.bytes(prmt(a0a, 0u, 0x4440u + l), a1a >> (7 * l));
                const uint2 eb = tab.bytes(prmt(a0b, 0u, 0x4440u + l), a1b >> (7 * l));
                const uint32_t x0 = xf[8 * sb + 2 * l], x1 = xf[8 * sb + 2 * l + 1];
                if (l == 0) imma0<true>(d, ea.x, eb.x, ea.y, eb.y, x0, x1);
                else imma<true>(d, ea.x, eb.x, ea.y, eb.y, x0, x1);
            }
            sum[sb][0] = join_hi_lo(d[0], d[1]);
            sum[sb][1] = join_hi_lo(d[2], d[3]);
        }
        const float sa0 = 0.5f + (float)(wa[1] >> 28), sa1 = 0.5f + (float)(wa[3] >> 28);
        const float sb0 = 0.5f + (float)(wb[1] >> 28), sb1 = 0.5f + (float)(wb[3] >> 28);
        acc[0] += (0.25f * xs * da) * (sa0 * sum[0][0] + sa1 * sum[1][0]);
        acc[1] += (0.25f * xs * db) * (sb0 * sum[0][1] + sb1 * sum[1][1]);
    }
}

// ---- staging x ------------------------------------------------------------------
// SEP: one column as a hi and a lo byte column.  An item is 8 consecutive k; the
// 32 items of a 256-wide unit are the 32 lanes of one warp, so the unit's largest
// magnitude is one warp reduction.  Magnitudes are compared as integers (the bit
// patterns of non-negative floats order like the floats, and every NaN pattern lies
// above infinity, so a NaN anywhere in the unit comes out on top and is seen).
// Rounding: v * inv + (1.5 * 2^23 + 128) lands where the float's low mantissa bits are
// the integer q + 128 = 256 * hi + (lo + 128): hi is byte 1, lo is byte 0 with its top
// bit flipped.  Byte order inside a quarter: k order (Q2_0: inside each 16, byte 4s + b
// holds k = s + 4b, the order the masked code words come in).  The quarter's record
// {scale, scale * sum of x over its first 32-wide block, over its second} follows its 64
// bytes in the first byte column.
template <int XDT> struct XRaw8 { uint4 v[XDT == DT_F32 ? 2 : 1]; };
template <int XDT>
__device__ __forceinline__ void x_floats(const XRaw8<XDT> &raw, float (&v)[8]) {
    if constexpr (XDT == DT_F32) {
        v[0] = __uint_as_float(raw.v[0].x); v[1] = __uint_as_float(raw.v[0].y);
        v[2] = __uint_as_float(raw.v[0].z); v[3] = __uint_as_float(raw.v[0].w);
        v[4] = __uint_as_float(raw.v[1].x); v[5] = __uint_as_float(raw.v[1].y);
        v[6] = __uint_as_float(raw.v[1].z); v[7] = __uint_as_float(raw.v[1].w);
    } else {
        const uint32_t w[4] = {raw.v[0].x, raw.v[0].y, raw.v[0].z, raw.v[0].w};
#pragma unroll
        for (int e = 0; e < 4; e++) {
            if constexpr (XDT == DT_F16) {
                const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&w[e]));
                v[2 * e] = f.x; v[2 * e + 1] = f.y;
            } else {
                v[2 * e] = __uint_as_float(w[e] << 16);
                v[2 * e + 1] = __uint_as_float(w[e] & 0xFFFF0000u);
            }
        }
    }
}

// The largest magnitude of a unit whose 32 items are in the lanes of a warp; a NaN if there is one (every NaN's bits lie
// above infinity's).
__device__ __forceinline__ float unit_max(const float (&v)[8]) {
    auto top = [](float a, float b) {
        float m;
        asm("max.NaN.f32 %0, %1, %2;" : "=f"(m) : "f"(fabsf(a)), "f"(fabsf(b)));
        return m;
    };
    const float m = top(top(top(v[0], v[1]), top(v[2], v[3])), top(top(v[4], v[5]), top(v[6], v[7])));
    return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(m) & 0x7FFFFFFFu));
}

template <int TY, int XDT, uint32_t NW = kGemvWarps>
__device__ __forceinline__ void stage_x_bytes(uint32_t xs32, uint32_t es, const void *x, uint32_t u_first, uint32_t nu,
                                              uint32_t tid) {
    const uint32_t items = nu * 32;
    constexpr uint32_t kFlight = 4;  // items a thread has in flight: the loads go out first
    constexpr uint32_t kMagicBits = 0x4B400080u;  // 1.5 * 2^23 + 128 as a float
    const uint32_t e8 = tid & 31;  // this lane's item inside its unit, the same in every pass
    // Its quarter, and which half of that its 32-wide block is.  Q6_K: thread 2h + s takes blocks 4h + s and 4h + s + 2.
    const uint32_t c = TY == T_Q6_K ? (e8 >> 4) * 2 + ((e8 >> 2) & 1) : e8 >> 3;
    const uint32_t second = TY == T_Q6_K ? (e8 >> 3) & 1 : (e8 >> 2) & 1;
    const uint32_t item_off = c * kSepQuarter + second * 32 + (e8 & 3) * 8;  // 8 bytes of the quarter's 64
    for (uint32_t base = tid; base < items; base += kFlight * NW * 32) {
        XRaw8<XDT> raw[kFlight];
#pragma unroll
        for (uint32_t r = 0; r < kFlight; r++) {
            const uint32_t i = base + r * NW * 32;
            const uint4 *src = reinterpret_cast<const uint4 *>(reinterpret_cast<const uint8_t *>(x) +
                                                              ((size_t)u_first * 256 + (size_t)i * 8) * (XDT == DT_F32 ? 4 : 2));
#pragma unroll
            for (int j = 0; j < (XDT == DT_F32 ? 2 : 1); j++)
                raw[r].v[j] = i < items ? ld_dep(src + j) : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (uint32_t r = 0; r < kFlight; r++) {
            const uint32_t i = base + r * NW * 32;
            if (i >= items) break;  // the same for the whole warp: a warp holds one unit
            float v[8];
            x_floats<XDT>(raw[r], v);
            const float amax = unit_max(v);
            // amax below 1e-30: the unit counts as zeros (32512 / amax would overflow, and its
            // products vanish in fp32 anyway); amax infinite: inv = 0, scale = inf; amax a NaN:
            // both comparisons fail, inv = 0, and the scale is that NaN
            const float inv = amax > 1e-30f ? __fdividef(kXqMax, amax) : 0.f;
            const float scale = amax * (1.f / kXqMax);
            uint32_t t[8], tsum = 0;
#pragma unroll
            for (int j = 0; j < 8; j++) {
                t[j] = __float_as_uint(fmaf(v[j], inv, __uint_as_float(kMagicBits)));
                tsum += t[j];
            }
            int qsum = (int)(tsum - 8u * kMagicBits);  // sum of the eight q
            qsum += __shfl_xor_sync(0xffffffffu, qsum, 1);
            // Q6_K: the sums over 16-wide groups, in the second byte column
            if constexpr (TY == T_Q6_K)
                if ((e8 & 1) == 0) sts32(xs32 + es + (i >> 5) * kSepUnit + c * kSepQuarter + 64 + second * 8 + (e8 & 2) * 2, __float_as_uint(scale * (float)qsum));
            qsum += __shfl_xor_sync(0xffffffffu, qsum, 2);
            const uint32_t u = i >> 5;
            const uint32_t dst = xs32 + u * kSepUnit + item_off;
            if constexpr (TY == T_Q2_0) {
                // this item is half (e8 & 1) of a 16: bytes 2h, 2h + 1 of each of its four words
                const uint32_t at16 = dst - (e8 & 1) * 8;
#pragma unroll
                for (int w = 0; w < 4; w++) {
                    const uint32_t at = at16 + 4 * w + 2 * (e8 & 1);
                    sts16(at, prmt(t[w], t[w + 4], 0x0051u) & 0xFFFFu);
                    sts16(at + es, (prmt(t[w], t[w + 4], 0x0040u) & 0xFFFFu) ^ 0x8080u);
                }
            } else {
                const uint32_t h0 = prmt(prmt(t[0], t[1], 0x0051u), prmt(t[2], t[3], 0x0051u), 0x5410u);
                const uint32_t h1 = prmt(prmt(t[4], t[5], 0x0051u), prmt(t[6], t[7], 0x0051u), 0x5410u);
                const uint32_t l0 = prmt(prmt(t[0], t[1], 0x0040u), prmt(t[2], t[3], 0x0040u), 0x5410u) ^ 0x80808080u;
                const uint32_t l1 = prmt(prmt(t[4], t[5], 0x0040u), prmt(t[6], t[7], 0x0040u), 0x5410u) ^ 0x80808080u;
                if constexpr (TY == T_IQ4_NL) {
                    // k 4i, 16+4i, 4i+1, 17+4i, then 4i+2, ...: the item 16 k further on, or back, is two lanes away
                    const bool high = e8 & 2;
                    const uint32_t at = xs32 + u * kSepUnit + c * kSepQuarter + (e8 & 4) * 8 + (e8 & 1) * 16 + (e8 & 2) * 4;
                    const uint32_t hx = __shfl_xor_sync(0xffffffffu, high ? h0 : h1, 2), lx = __shfl_xor_sync(0xffffffffu, high ? l0 : l1, 2);
                    const uint32_t ha = high ? hx : h0, hb = high ? h1 : hx, la = high ? lx : l0, lb = high ? l1 : lx;
                    sts64(at, prmt(ha, hb, 0x5140u), prmt(ha, hb, 0x7362u));
                    sts64(at + es, prmt(la, lb, 0x5140u), prmt(la, lb, 0x7362u));
                } else {
                    sts64(dst, h0, h1);
                    sts64(dst + es, l0, l1);
                }
            }
            // the quarter's record, behind its 64 bytes in the first byte column
            const uint32_t rec = xs32 + u * kSepUnit + c * kSepQuarter + 64;
            if ((e8 & 3) == 0 && !second) sts32(rec, __float_as_uint(scale));
            if ((e8 & 3) == 0) sts32(rec + 4 + second * 4, __float_as_uint(scale * (float)qsum));
        }
    }
}

// WIDE: every column as two to four byte columns of the panel, `es` bytes from one to the next.  An item is 8 consecutive k; the 32 items of a (column, unit)
// pair are the lanes of one warp.  Two bytes: the integers of the one-column panel.  Three and four: v = q * 2^-s, |q| <=
// 2^22 and 2^30, s from the largest magnitude's exponent and at most 149, so that the scale is a float however
// small x is.  Inside a unit of a byte column thread c's 64 bytes start at 64c: eight bytes per
// 32-wide block in the type's WideOrder, block after block, the 16-byte pieces of threads 2 and 3
// swapped in pairs (see kXqUnit).
template <int TY, int MODE, int XDT, uint32_t NW = kGemvWarps>
__device__ __forceinline__ void stage_x_wide(uint32_t xs32, uint32_t es, uint32_t info32, const void *x, uint32_t kdim, uint32_t ncols,
                                             uint32_t u_first, uint32_t nu, uint32_t tid) {
    using W = WideMode<MODE>;
    constexpr int NB = W::nb;
    constexpr uint32_t IW = wide_info_words(TY, NB);
    const uint32_t warp = __shfl_sync(0xffffffffu, tid >> 5, 0), e8 = tid & 31, blk = e8 >> 2, e4 = e8 & 3;
    const uint32_t pairs = ncols * nu;
    if (pairs == 0) return;
    constexpr uint32_t kFlight = 4;
    constexpr uint32_t kMagicBits = 0x4B400080u;  // 1.5 * 2^23 + 128 as a float
    constexpr uint32_t ES = XDT == DT_F32 ? 4 : 2, UX = 256 * ES;
    // The (column, unit) pairs, unit by unit and column after column, in a run a warp: addresses move by constants.
    const uint32_t lo = pairs * warp / NW, hi = pairs * (warp + 1) / NW, col0 = lo / nu;
    uint32_t lu = lo - col0 * nu, su = lu;  // units of what is loaded and of what is stored next
    const uint8_t *src = reinterpret_cast<const uint8_t *>(x) + (size_t)col0 * (kdim * ES) + (size_t)(u_first + lu) * UX + e8 * (8 * ES);
    const uint32_t wrap = kdim * ES - nu * UX;  // (mod 2^32; added as a signed number)
    uint32_t dst0 = xs32 + col0 * NB * es + su * kXqUnit, info0 = info32 + (su * ncols + col0) * (IW * 4);
    for (uint32_t base = lo; base < hi; base += kFlight) {
        XRaw8<XDT> raw[kFlight];
#pragma unroll
        for (uint32_t r = 0; r < kFlight; r++) {
            const bool live = base + r < hi && (!W::rag || (u_first + lu) * 256 + e8 * 8 < kdim);
#pragma unroll
            for (int j = 0; j < (XDT == DT_F32 ? 2 : 1); j++)
                raw[r].v[j] = live ? ld_dep(reinterpret_cast<const uint4 *>(src) + j) : make_uint4(0u, 0u, 0u, 0u);
            src += UX;
            if (++lu == nu) {
                lu = 0;
                src += (int32_t)wrap;
            }
        }
#pragma unroll
        for (uint32_t r = 0; r < kFlight; r++) {
            if (base + r >= hi) break;  // the same for the whole warp
            float v[8];
            x_floats<XDT>(raw[r], v);
            const float amax = unit_max(v);
            const uint32_t mb = __float_as_uint(amax);
            // as in the one-column panel: below 1e-30 the unit counts as zeros, an infinite
            // amax gives inv = 0 and an infinite scale, a NaN gives inv = 0 and a NaN scale
            float scale;
            uint32_t w[NB][2];  // [byte][first, second four k]
            if constexpr (NB == 2) {
                const float inv = amax > 1e-30f ? __fdividef(kXqMax, amax) : 0.f;
                scale = amax * (1.f / kXqMax);
                uint32_t t[8];
#pragma unroll
                for (int j = 0; j < 8; j++) t[j] = __float_as_uint(fmaf(v[j], inv, __uint_as_float(kMagicBits)));
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    w[0][i] = prmt(prmt(t[4 * i], t[4 * i + 1], 0x0051u), prmt(t[4 * i + 2], t[4 * i + 3], 0x0051u), 0x5410u);
                    w[1][i] = prmt(prmt(t[4 * i], t[4 * i + 1], 0x0040u), prmt(t[4 * i + 2], t[4 * i + 3], 0x0040u), 0x5410u) ^ 0x80808080u;
                }
            } else {
                // An infinity counts as its sign and everything else as zero, with an infinite scale: the sums
                // come out as the infinity or NaN that fp32 products give.  A NaN: a NaN scale.
                const bool finite = mb < 0x7F800000u;
                const int sh = finite ? (NB == 4 ? 156 - (int)max(mb >> 23, 7u) : 148 - (int)max(mb >> 23, 1u)) : 0;
                scale = !finite ? amax : __uint_as_float(sh <= 126 ? (uint32_t)(127 - sh) << 23 : 1u << (149 - sh));
                // 2^sh in two factors: it may be beyond the largest float
                const float f1 = __uint_as_float((uint32_t)(127 + (sh >> 1)) << 23), f2 = __uint_as_float((uint32_t)(127 + sh - (sh >> 1)) << 23);
                uint32_t t[8];
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const float f = finite ? v[j] * f1 * f2 : isinf(v[j]) ? copysignf(1.f, v[j]) : 0.f;
                    t[j] = (uint32_t)__float2int_rn(f) + (NB == 4 ? 0x808080u : 0x8080u);
                }
#pragma unroll
                for (int i = 0; i < 2; i++)
#pragma unroll
                    for (int b = 0; b < NB; b++) {
                        const uint32_t sel = 0x0040u + 0x0011u * (NB - 1 - b);  // byte NB - 1 - b of two words
                        w[b][i] = prmt(prmt(t[4 * i], t[4 * i + 1], sel), prmt(t[4 * i + 2], t[4 * i + 3], sel), 0x5410u) ^ (b ? 0x80808080u : 0u);
                    }
            }
            const uint32_t info = info0;
            if (e8 == 0) sts32(info, __float_as_uint(scale));
            int sums[NB];
#pragma unroll
            for (int b = 0; b < NB; b++) {
                const uint32_t dst = dst0 + b * es, at = blk & 1 ? 8 : 0;
                if constexpr (kWideOrder<TY> == O_SEQ) {
                    sts64(dst + xq_piece_offset(e4, blk >> 1) + at, w[b][0], w[b][1]);
                } else if constexpr (kWideOrder<TY> == O_SPLIT) {
#pragma unroll
                    for (int i = 0; i < 2; i++)
                        sts32(dst + xq_piece_offset(2 * (e4 & 1) + i, blk >> 1) + at + (e4 & 2) * 2, w[b][i]);
                } else if constexpr (kWideOrder<TY> == O_PAIRS) {
                    // the item 16 k further on, or back, is two lanes away
                    const uint32_t give = e4 & 2 ? w[b][0] : w[b][1], own = e4 & 2 ? w[b][1] : w[b][0];
                    const uint32_t got = __shfl_xor_sync(0xffffffffu, give, 2);
                    const uint32_t lo = e4 & 2 ? got : own, hi = e4 & 2 ? own : got;
                    sts64(dst + xq_piece_offset(2 * (e4 & 1) + (e4 >> 1), blk >> 1) + at, prmt(lo, hi, 0x5140u), prmt(lo, hi, 0x7362u));
                } else {
#pragma unroll
                    for (int c = 0; c < 4; c++)
                        sts16(dst + xq_piece_offset(c, blk >> 1) + at + (e4 >> 1) * 4 + (e4 & 1) * 2, prmt(w[b][0], w[b][1], (uint32_t)(c | (4 + c) << 4)) & 0xFFFFu);
                }
                sums[b] = __dp4a((int)w[b][0], 0x01010101, __dp4a((int)w[b][1], 0x01010101, 0));
            }
            if constexpr (TY == T_Q2_0) {
#pragma unroll
                for (int b = 0; b < NB; b++) {
#pragma unroll
                    for (int o = 1; o < 16; o <<= 1) sums[b] += __shfl_xor_sync(0xffffffffu, sums[b], o);
                    if ((e8 & 15) == 0) sts32(info + 4 + ((e8 >> 4) * NB + b) * 4, (uint32_t)-sums[b]);
                }
            } else if constexpr (IW > 1) {
                constexpr uint32_t groups = TY == T_Q6_K ? 16 : 8;
                int sum = sums[0] * 256 + sums[1];
                sum += __shfl_xor_sync(0xffffffffu, sum, 1);
                if constexpr (TY != T_Q6_K) sum += __shfl_xor_sync(0xffffffffu, sum, 2);
                if ((e8 & (32 / groups - 1)) == 0) {
                    const uint32_t t = (uint32_t)(sum + 0x8080), g = e8 / (32 / groups);
                    sts8(info + 4 + g, t >> 16);
                    sts8(info + 4 + groups + g, (t >> 8 & 255u) ^ 0x80u);
                    sts8(info + 4 + 2 * groups + g, (t & 255u) ^ 0x80u);
                }
            }
            dst0 += kXqUnit;
            info0 += ncols * (IW * 4);
            if (++su == nu) {
                su = 0;
                dst0 += NB * es - nu * kXqUnit;
                info0 += IW * 4 - pairs * (IW * 4);
            }
        }
    }
}

}  // namespace okf
