// The decode matvec's arithmetic for several activation columns ("WIDE").
//
// Weights are the A operand of the integer MMA (16 output rows), bytes of x the B operand, in one or
// two sets of eight byte columns.  A column of x is two signed bytes per element (q = 256 * hi + lo,
// 16 bits), or three or four for rows that are no multiple of 256 weights, whose scale is a power of two.
// (Those shapes ran on fp32 arithmetic before there was a kernel for them and keep that precision: 31 bits
// hold an fp32 x exactly down to 2^-7 of the unit's largest, 23 bits an fp16 x down to 2^-11 and a bf16 x to 2^-14 of
// it.  With 24 bits and a scale of any value, results of fp32 x were 1.2 to 1.6 times as far from float64 as fp32
// sums on rows up to 2000 weights.  Four bytes for 16-bit x too: Q4_0 8224 -> 6000, 4 columns, 22.7 -> 30.3 us,
// as less of x fits beside the ring.)
//   W1  up to 4 columns: byte column 2j = hi, 2j + 1 = lo of column j
//   W2  up to 8 columns: the same for columns 4 .. 7 in a second set.  Weights are unpacked and
//       scales decoded once for both (before, eight columns were two launches over the weights)
//   R4  up to 4 columns of four bytes (fp32 x): the upper two in the first set, the lower two in the second
//   R3  up to 4 columns of three bytes (16-bit x): hi and mid in the first set, lo in column 2j of the second
// Thread (g = lane / 4, c = lane % 4) feeds output rows g and g + 8 at k-slots 4c .. 4c+3 and 16+4c ..
// of a block, byte column g at the same slots, and gets back, for its own two rows, column c (and
// 4 + c): all bytes of a column meet in one thread.  (With x as the A operand instead, 8 output rows
// per MMA, the operand quads had to be put together by register moves and every thread decoded the
// scales of two other rows: Q4_K 2560 -> 19456, 4 columns, 18.3 us against 12.5.)
//
// Which real k a slot stands for is free as long as both operands agree; each type has the order in
// which its weights lie in memory (kWideOrder).
#pragma once
#include "okf_gemv_mma.cuh"

namespace okf {

enum : int { M_SEP = 0, M_W1 = 1, M_W2 = 2, M_R4 = 3, M_R3 = 4 };
// bytes of an element of x
__host__ __device__ constexpr int mode_bytes(int mode) { return mode == M_R4 ? 4 : mode == M_R3 ? 3 : 2; }
template <int MODE> struct WideMode {
    static constexpr int sets = MODE == M_W2 || mode_bytes(MODE) > 2 ? 2 : 1;  // sets of eight byte columns
    static constexpr int nb = mode_bytes(MODE);                    // bytes per element
    static constexpr int vals = MODE == M_W2 ? 2 : 1;                 // columns of a thread
    static constexpr bool rag = nb > 2;                             // rows end inside a unit, 2-byte aligned
};

// Order of a block's 32 k over the threads' slots (thread c's eight bytes, first word then second):
//   seq    k 8c .. 8c+7
//   split  k 4c .. 4c+3, 16+4c .. 16+4c+3      (both nibbles of a byte; both 16-wide scale groups)
//   pairs  k 4c, 16+4c, 4c+1, 17+4c, then +2   (IQ4_NL: nibbles as they follow in a word)
//   comb   k 4b+c, then 16+4b+c, b = 0 .. 3    (Q2_0: code c of every byte)
enum : int { O_SEQ, O_SPLIT, O_PAIRS, O_COMB };
template <int TY> constexpr int kWideOrder = TY == T_Q4_0 || TY == T_Q6_K ? O_SPLIT : TY == T_IQ4_NL ? O_PAIRS : TY == T_Q2_0 ? O_COMB : O_SEQ;

// What lies beside a column's bytes in a unit, in words: its scale and, for types with an offset, sums
// of x.  Q4_K and Q5_K over the eight blocks, Q6_K over the sixteen 16-wide groups, as three bytes
// s = 65536 * s2 + 256 * s1 + s0, plane after plane (s2, s1, s0); Q2_0 over the two 128-wide blocks,
// negated, one integer for every byte of x.
constexpr uint32_t wide_info_words(int ty, int nb) {
    return ty == T_Q4_K || ty == T_Q5_K ? 7u : ty == T_Q6_K ? 13u : ty == T_Q2_0 ? 1u + 2u * nb : 1u;
}

// D (16 x 8) = A * B + C; a: rows g, g + 8 in the first word of slots, then in the second
template <bool SIGNED_A>
__device__ __forceinline__ void wmma32(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1, int c0,
                                       int c1, int c2, int c3) {
    if constexpr (SIGNED_A)
        asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
            : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(c0), "r"(c1), "r"(c2), "r"(c3));
    else
        asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
            : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(c0), "r"(c1), "r"(c2), "r"(c3));
}
template <bool SIGNED_A, bool SIGNED_B>
__device__ __forceinline__ void wmma16(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    if constexpr (SIGNED_A && SIGNED_B)
        asm("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
            : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a0), "r"(a1), "r"(b0), "r"(0));
    else
        asm("mma.sync.aligned.m16n8k16.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
            : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a0), "r"(a1), "r"(b0), "r"(0));
}

// What a thread holds of x for one unit.
template <int TY, int MODE> struct WideX {
    using W = WideMode<MODE>;
    uint32_t f[W::sets][16];  // block b of byte column g: f[.][2b], f[.][2b + 1]
    float scale[W::vals];     // of this thread's columns
    // Q4_K, Q5_K, Q6_K: B operands of the offsets' two MMAs per set; Q2_0: [block][byte] of this thread's columns
    uint32_t sum[W::vals][TY == T_Q2_0 ? 2 * W::nb : 2];
    template <bool SA> __device__ __forceinline__ void mma(int (&d)[W::sets][4], int b, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3) const {
#pragma unroll
        for (int s = 0; s < W::sets; s++) wmma32<SA>(d[s], a0, a1, a2, a3, f[s][2 * b], f[s][2 * b + 1], 0, 0, 0, 0);
    }
    template <bool SA> __device__ __forceinline__ void mma_on(int (&d)[W::sets][4], int b, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3) const {
#pragma unroll
        for (int s = 0; s < W::sets; s++)
            wmma32<SA>(d[s], a0, a1, a2, a3, f[s][2 * b], f[s][2 * b + 1], d[s][0], d[s][1], d[s][2], d[s][3]);
    }
    // offsets of rows g, g + 8 (bytes of w0, w1 in slots 0 .. 15) times the sums of x
    template <bool SA> __device__ __forceinline__ void offsets(int (&m)[W::vals][2], uint32_t w0, uint32_t w1) const {
#pragma unroll
        for (int s = 0; s < W::vals; s++) {
            int hi[4], lo[4];
            wmma16<SA, true>(hi, w0, w1, sum[s][0]);  // columns 2c: s2, 2c + 1: s1
            wmma16<SA, true>(lo, w0, w1, sum[s][1]);  // columns 2c: s0
            m[s][0] = (hi[0] * 256 + hi[1]) * 256 + lo[0];
            m[s][1] = (hi[2] * 256 + hi[3]) * 256 + lo[2];
        }
    }
};

// The bytes of a column put together: v[column][row].  FITS: 256 * hi + lo does not leave 32 bits.
template <int MODE, bool FITS>
__device__ __forceinline__ void wide_join(const int (&d)[WideMode<MODE>::sets][4], float (&v)[WideMode<MODE>::vals][2]) {
    using W = WideMode<MODE>;
#pragma unroll
    for (int r = 0; r < 2; r++) {
        if constexpr (W::nb == 4) {
            v[0][r] = fmaf((float)(d[0][2 * r] * 256 + d[0][2 * r + 1]), 65536.f, (float)(d[W::sets - 1][2 * r] * 256 + d[W::sets - 1][2 * r + 1]));
        } else if constexpr (W::nb == 3) {
            v[0][r] = fmaf((float)d[0][2 * r], 65536.f, (float)(d[0][2 * r + 1] * 256 + d[W::sets - 1][2 * r]));
        } else {
#pragma unroll
            for (int s = 0; s < W::vals; s++)
                v[s][r] = FITS ? (float)(d[s][2 * r] * 256 + d[s][2 * r + 1]) : fmaf((float)d[s][2 * r], 256.f, (float)d[s][2 * r + 1]);
        }
    }
}

// IQ2_XXS look-ups.  A codebook entry is eight magnitudes out of {8, 25, 43}; in shared memory it is
// eight 4-bit selectors of a byte permute over {8, 25, 43, 0, -8, -25, -43, 0}, one word, and a 7-bit
// sign index (its eighth sign is the parity of the seven, LLM/Quantize/IQ2Grid.swift:73-85) the
// selector bits that pick the negative half.  Two one-word look-ups and an OR give the eight signed
// bytes in two permutes.  (Before: a 64-bit look-up, the signs' byte masks worked out with popc,
// multiplies and permutes, XORs, and a second MMA over the masks.)  Both tables hold every entry
// `copies` times side by side, lane l reads copy l mod copies: 32 copies make every access free of
// bank conflicts.
constexpr uint32_t kIq2Pos = 0x002B1908u, kIq2Neg = 0x00D5E7F8u;
__host__ __device__ constexpr uint32_t iq2_code_selectors(uint64_t entry) {
    uint32_t s = 0;
#pragma unroll
    for (int j = 0; j < 8; j++) s |= (uint32_t)(entry >> (8 * j + 4) & 3u) << (4 * j);  // 8, 25, 43 -> 0, 1, 2
    return s;
}
__host__ __device__ constexpr uint32_t iq2_sign_selectors(uint32_t idx7) {
    const uint32_t a = idx7 ^ idx7 >> 4, b = a ^ a >> 2;
    uint32_t s = ((b ^ b >> 1) & 1u) << 30;
#pragma unroll
    for (int j = 0; j < 7; j++) s |= (idx7 >> j & 1u) << (4 * j + 2);
    return s;
}
// both tables, worked out by the compiler: 256 codes, then 128 signs (for okf_gemv_stream.cu; in the other kernels, whose threads have an entry or two
// each to work out, loads of these made launches 0.1 to 0.3 % longer)
struct Iq2Selectors {
    uint32_t v[384];
    constexpr Iq2Selectors() : v{} {
        constexpr uint64_t grid[256] = {OKF_IQ2XXS_GRID_VALUES};
        for (uint32_t i = 0; i < 256; i++) v[i] = iq2_code_selectors(grid[i]);
        for (uint32_t i = 0; i < 128; i++) v[256 + i] = iq2_sign_selectors(i);
    }
};
static __device__ constexpr Iq2Selectors g_iq2_selectors;
struct Iq2Tab {
    uint32_t code, sign;  // shared addresses of this lane's copy of entry 0
    uint32_t stride;      // bytes between entries
    __device__ __forceinline__ uint2 bytes(uint32_t index, uint32_t signs) const {
        const uint32_t s = lds32(code + index * stride) | lds32(sign + (signs & 127u) * stride);
        return make_uint2(prmt(kIq2Pos, kIq2Neg, s), prmt(kIq2Pos, kIq2Neg, s >> 16));
    }
};

// IQ4_NL: the sixteen codebook values (LLM/Gemma/Gemma4Quant.swift:5-9) for the eight nibbles of a
// word, in the order the nibbles follow (lo, hi of byte 0, lo, hi of byte 1, ...): a nibble's low
// three bits are a permute selector as they stand, once into the low half of the table and once into
// the high half; bit 3, moved to bit 2 of a third selector, picks between the two.
__device__ __forceinline__ uint2 iq4nl_word(uint32_t w) {
    // {-127, -104, -83, -65}, {-49, -35, -22, -10}, {1, 13, 25, 38}, {53, 69, 89, 113}
    constexpr uint32_t T0 = 0xBFAD9881u, T1 = 0xF6EADDCFu, T2 = 0x26190D01u, T3 = 0x71594535u;
    const uint32_t sel = w & 0x77777777u, pick = (w >> 1 & 0x44444444u) | 0x32103210u;
    uint2 r;
    r.x = prmt(prmt(T0, T1, sel), prmt(T2, T3, sel), pick);
    r.y = prmt(prmt(T0, T1, sel >> 16), prmt(T2, T3, sel >> 16), pick >> 16);
    return r;
}

// Words of a row at a 2-byte aligned shared address.  Where they start inside an aligned word is worked out once
// for all of them (anew for every few words: IQ2_XXS 5120 -> 17408 twice, 4 columns, 36.4 us, so 34.1).
struct RowA2 {
    uint32_t base, sh;
    __device__ __forceinline__ explicit RowA2(uint32_t a) : base(a & ~3u), sh((a & 2u) * 8u) {}
    // 4 * NW bytes `off` (a multiple of four) behind the start
    template <int NW> __device__ __forceinline__ void get(uint32_t off, uint32_t (&out)[NW]) const {
        uint32_t w[NW + 1];
#pragma unroll
        for (int i = 0; i <= NW; i++) w[i] = lds32(base + off + 4 * i);
#pragma unroll
        for (int i = 0; i < NW; i++) out[i] = __funnelshift_r(w[i], w[i + 1], sh);
    }
    __device__ __forceinline__ uint32_t word(uint32_t off) const {
        uint32_t v[1];
        get<1>(off, v);
        return v[0];
    }
};

// One unit of sixteen output rows.  ua, ub: shared addresses of the unit in rows g and g + 8.  left:
// blocks of 32 weights the row still has from this unit on (R only; those past the end hold the next
// row's bytes against zeros of x, and may look like infinite scales).  acc[column][row].
template <int TY, int MODE>
__device__ __forceinline__ void unit_wide(uint32_t ua, uint32_t ub, uint32_t c, const WideX<TY, MODE> &X, const Iq2Tab &tab, uint32_t left,
                                          float (&acc)[WideMode<MODE>::vals][2]) {
    using W = WideMode<MODE>;
    constexpr int NV = W::vals, NS = W::sets;
    constexpr bool RAG = W::rag;
    float sum[NV][2];  // of the unit, in units of x's scale
#pragma unroll
    for (int i = 0; i < NV; i++) sum[i][0] = sum[i][1] = 0.f;
    constexpr uint32_t ml = 0x0F0F0F0Fu;

    if constexpr (TY == T_Q4_K || TY == T_Q5_K) {
        // {f16 d; f16 dmin; u8 scales[12]; [Q5_K: u8 qh[32];] u8 qs[128]} (LLM/Quantize/KQuants.swift:104-158).
        // 32 bytes of qs: block 2p in the low nibbles, 2p + 1 in the high ones; bit j of qh[l] is the
        // fifth bit of block j.  Block sums are multiplied by their 6-bit scales as integers.
        const uint4 ha = lds128(ua), hb = lds128(ub);
        const uint32_t a03 = ha.y & 0x3F3F3F3Fu, a47 = (ha.w & ml) | ((ha.y >> 2) & 0x30303030u);
        const uint32_t b03 = hb.y & 0x3F3F3F3Fu, b47 = (hb.w & ml) | ((hb.y >> 2) & 0x30303030u);
        uint2 ga = make_uint2(0u, 0u), gb = ga;
        if constexpr (TY == T_Q5_K) {
            ga = lds64(ua + 16 + 8 * c);
            gb = lds64(ub + 16 + 8 * c);
        }
        int te[NS][4], to[NS][4];  // scale * block sum: low-nibble / high-nibble blocks
#pragma unroll
        for (int p = 0; p < 4; p++) {
            const uint2 wa = lds64(ua + (TY == T_Q5_K ? 48 : 16) + 32 * p + 8 * c), wb = lds64(ub + (TY == T_Q5_K ? 48 : 16) + 32 * p + 8 * c);
            const uint32_t sa = p < 2 ? a03 : a47, sb = p < 2 ? b03 : b47;
            auto bit = [](uint32_t v, int j) { return (j < 4 ? v << (4 - j) : v >> (j - 4)) & 0x10101010u; };
            int d[NS][4];
            const int ea = ubyte(sa, (2 * p) & 3), eb = ubyte(sb, (2 * p) & 3);
            if constexpr (TY == T_Q4_K) X.template mma<false>(d, 2 * p, wa.x & ml, wb.x & ml, wa.y & ml, wb.y & ml);
            else X.template mma<false>(d, 2 * p, (wa.x & ml) | bit(ga.x, 2 * p), (wb.x & ml) | bit(gb.x, 2 * p), (wa.y & ml) | bit(ga.y, 2 * p),
                                       (wb.y & ml) | bit(gb.y, 2 * p));
#pragma unroll
            for (int s = 0; s < NS; s++)
#pragma unroll
                for (int e = 0; e < 4; e++) te[s][e] = (e < 2 ? ea : eb) * d[s][e] + (p ? te[s][e] : 0);
            const int oa = ubyte(sa, (2 * p + 1) & 3), ob = ubyte(sb, (2 * p + 1) & 3);
            if constexpr (TY == T_Q4_K) {  // left where they are: 16 x the value, taken out of the sums
                constexpr uint32_t mh = 0xF0F0F0F0u;
                X.template mma<false>(d, 2 * p + 1, wa.x & mh, wb.x & mh, wa.y & mh, wb.y & mh);
            } else {
                X.template mma<false>(d, 2 * p + 1, (wa.x >> 4 & ml) | bit(ga.x, 2 * p + 1), (wb.x >> 4 & ml) | bit(gb.x, 2 * p + 1),
                                      (wa.y >> 4 & ml) | bit(ga.y, 2 * p + 1), (wb.y >> 4 & ml) | bit(gb.y, 2 * p + 1));
            }
#pragma unroll
            for (int s = 0; s < NS; s++)
#pragma unroll
                for (int e = 0; e < 4; e++) to[s][e] = (e < 2 ? oa : ob) * d[s][e] + (p ? to[s][e] : 0);
        }
        // mins: an MMA of the rows' eight 6-bit mins with the sums of x over the blocks
        const uint32_t m03 = ha.z & 0x3F3F3F3Fu, m47 = ((ha.w >> 4) & ml) | ((ha.z >> 2) & 0x30303030u);
        const uint32_t n03 = hb.z & 0x3F3F3F3Fu, n47 = ((hb.w >> 4) & ml) | ((hb.z >> 2) & 0x30303030u);
        int mi[NV][2];
        X.template offsets<false>(mi, c == 0 ? m03 : c == 1 ? m47 : 0u, c == 0 ? n03 : c == 1 ? n47 : 0u);
#pragma unroll
        for (int s = 0; s < NS; s++)
#pragma unroll
            for (int e = 0; e < 4; e++) te[s][e] += TY == T_Q4_K ? to[s][e] >> 4 : to[s][e];  // exact multiples of 16
        float v[NV][2];
        wide_join<MODE, false>(te, v);
        const float2 fa = __half22float2(*reinterpret_cast<const __half2 *>(&ha.x)), fb = __half22float2(*reinterpret_cast<const __half2 *>(&hb.x));
#pragma unroll
        for (int i = 0; i < NV; i++) {
            sum[i][0] = fa.x * v[i][0] - fa.y * (float)mi[i][0];
            sum[i][1] = fb.x * v[i][1] - fb.y * (float)mi[i][1];
        }
    } else if constexpr (TY == T_Q6_K) {
        // {u8 ql[128]; u8 qh[64]; i8 scales[16]; f16 d} (LLM/Quantize/KQuants.swift:160-177): granule r of half n
        // has its low four bits in ql (byte 64n + 32(r & 1) + l, low nibble for r < 2), two more in qh, and a
        // scale per 16.  The codes go in unsigned; 32 x the sum of x leaves through the offsets' MMA.
        const RowA2 A(ua), B(ub), Ac(ua + 4 * c), Bc(ub + 4 * c);
        uint32_t sa[4], sb[4];
        A.get<4>(192, sa);
        B.get<4>(192, sb);
        auto sbyte = [](uint32_t v, int i) { return (int)prmt(v, 0u, 0x8880u + 0x1111u * i); };
        int te[NS][4];
#pragma unroll
        for (int n = 0; n < 2; n++) {
            uint32_t qa[4], qb[4], ha[2], hb[2];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                qa[i] = Ac.word(64 * n + 16 * i);
                qb[i] = Bc.word(64 * n + 16 * i);
            }
#pragma unroll
            for (int i = 0; i < 2; i++) {
                ha[i] = Ac.word(128 + 32 * n + 16 * i);
                hb[i] = Bc.word(128 + 32 * n + 16 * i);
            }
#pragma unroll
            for (int r = 0; r < 4; r++) {
#pragma unroll
                for (int i = 0; i < 2; i++) {  // the two 16-wide groups
                    auto code = [&](uint32_t q, uint32_t h) {
                        return ((r < 2 ? q : q >> 4) & ml) | ((r < 2 ? h << (4 - 2 * r) : h >> (2 * r - 4)) & 0x30303030u);
                    };
                    const uint32_t a0 = code(qa[2 * (r & 1) + i], ha[i]), a1 = code(qb[2 * (r & 1) + i], hb[i]);
                    const int blk = 4 * n + r, grp = 2 * blk + i;
                    const int ea = sbyte(sa[grp >> 2], grp & 3), eb = sbyte(sb[grp >> 2], grp & 3);
#pragma unroll
                    for (int s = 0; s < NS; s++) {
                        int d[4];
                        wmma16<false, true>(d, a0, a1, X.f[s][2 * blk + i]);
#pragma unroll
                        for (int e = 0; e < 4; e++) te[s][e] = (e < 2 ? ea : eb) * d[e] + (grp ? te[s][e] : 0);
                    }
                }
            }
        }
        int mi[NV][2];
        X.template offsets<true>(mi, Ac.word(192), Bc.word(192));
        float v[NV][2];
        wide_join<MODE, false>(te, v);
        const float da = f16bits(lds16(ua + 208)), db = f16bits(lds16(ub + 208));
#pragma unroll
        for (int i = 0; i < NV; i++) {
            sum[i][0] = da * fmaf((float)mi[i][0], -32.f, v[i][0]);
            sum[i][1] = db * fmaf((float)mi[i][1], -32.f, v[i][1]);
        }
    } else if constexpr (TY == T_Q2_0) {
        // two blocks {f16 d; u8 qs[32]}, weight = (code - 1) * d (LLM/Base/Quant.swift:2-25); minus the
        // block's sum of x is where the accumulators start
#pragma unroll
        for (int blk = 0; blk < 2; blk++) {
            int d[NS][4];
#pragma unroll
            for (int s = 0; s < NS; s++) {
                constexpr int last = W::nb - 1;
                const int h = (int)(RAG ? X.sum[0][W::nb * blk + 2 * s] : X.sum[RAG ? 0 : s % NV][W::nb * blk]);
                const int l = (int)(RAG ? (2 * s < last ? X.sum[0][W::nb * blk + (2 * s < last ? 2 * s + 1 : last)] : 0u)
                                        : X.sum[RAG ? 0 : s % NV][W::nb * blk + 1]);
                d[s][0] = d[s][2] = h;
                d[s][1] = d[s][3] = l;
            }
            uint32_t wa[8], wb[8];
            if constexpr (RAG) {
                lds_a2<8>(ua + 34 * blk + 2, wa);
                lds_a2<8>(ub + 34 * blk + 2, wb);
            } else {  // units start on 4-byte boundaries
                const uint32_t at = 34 * blk + 2 - (blk ? 0 : 2);
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    uint32_t w[9];
#pragma unroll
                    for (int i = 0; i < (blk ? 8 : 9); i++) w[i] = lds32((r ? ub : ua) + at + 4 * i);
#pragma unroll
                    for (int i = 0; i < 8; i++) (r ? wb : wa)[i] = blk ? w[i] : __funnelshift_r(w[i], w[i + 1], 16);
                }
            }
#pragma unroll
            for (int b = 0; b < 4; b++) {  // 8 bytes = 32 codes; this thread takes code c of every byte
                constexpr uint32_t m = 0x03030303u;
                X.template mma_on<false>(d, 4 * blk + b, wa[2 * b] >> (2 * c) & m, wb[2 * b] >> (2 * c) & m, wa[2 * b + 1] >> (2 * c) & m,
                                         wb[2 * b + 1] >> (2 * c) & m);
            }
            float v[NV][2];
            wide_join<MODE, true>(d, v);
            float da = f16bits(lds16(ua + 34 * blk)), db = f16bits(lds16(ub + 34 * blk));
            if (RAG && 4u * blk >= left) da = db = 0.f;
#pragma unroll
            for (int i = 0; i < NV; i++) {
                sum[i][0] = fmaf(da, v[i][0], sum[i][0]);
                sum[i][1] = fmaf(db, v[i][1], sum[i][1]);
            }
        }
    } else if constexpr (TY == T_IQ2_XXS) {
        // {f16 d; 8 x (u32: four codebook indices, u32: four 7-bit sign indices + 4-bit scale)}
        // (LLM/Quantize/IQ2XXS.swift:34-53): entry c of every sub-block is this thread's eight weights.
        // Scale (0.5 + s) / 4 = (2s + 1) / 8 multiplies the integer sums.
        const RowA2 A(ua + 2), B(ub + 2);
        int te[NS][4];
#pragma unroll
        for (int b = 0; b < 8; b++) {
            // (index bytes by loads of their own: out of the words, with a funnel shift and a byte permute more on the fullest pipe, 5120 -> 2 x 17408, 4
            // columns, 30.7 us)
            const uint32_t ia = lds8(ua + 2 + 8 * b + c), ib = lds8(ub + 2 + 8 * b + c);
            const uint32_t wa = A.word(8 * b + 4), wb = B.word(8 * b + 4);
            const uint2 va = tab.bytes(ia, wa >> (7 * c)), vb = tab.bytes(ib, wb >> (7 * c));
            int d[NS][4];
            X.template mma<true>(d, b, va.x, vb.x, va.y, vb.y);
            const int ea = (int)(wa >> 27 | 1u), eb = (int)(wb >> 27 | 1u);  // 2 * (the upper four bits) + 1
#pragma unroll
            for (int s = 0; s < NS; s++)
#pragma unroll
                for (int e = 0; e < 4; e++) te[s][e] = (e < 2 ? ea : eb) * d[s][e] + (b ? te[s][e] : 0);
        }
        float v[NV][2];
        wide_join<MODE, false>(te, v);
        const float da = 0.125f * f16bits(lds16(ua)), db = 0.125f * f16bits(lds16(ub));
#pragma unroll
        for (int i = 0; i < NV; i++) {
            sum[i][0] = da * v[i][0];
            sum[i][1] = db * v[i][1];
        }
    } else {
        // eight blocks {f16 d; ...} of 32: Q8_0 i8 q[32] (LLM/Gemma/Gemma4Quant.swift:51-69), Q4_0 and IQ4_NL
        // u8 qs[16], byte j = weights j (low nibble) and j + 16 (:5-49).  Units whose rows are whole start on
        // 16-byte boundaries, so which words straddle is known at compile time.
        constexpr uint32_t BB = TY == T_Q8_0 ? 34 : 18;
#pragma unroll
        for (int b = 0; b < 8; b++) {
            uint32_t w[2][2];  // [row][word of slots]
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const uint32_t at = (r ? ub : ua) + BB * b + 2;
                if constexpr (TY == T_Q8_0) {
                    if constexpr (RAG) {
                        lds_a2<2>(at + 8 * c, w[r]);
                    } else if (b & 1) {
                        w[r][0] = lds32(at + 8 * c);
                        w[r][1] = lds32(at + 8 * c + 4);
                    } else {
                        const uint32_t w0 = lds32(at + 8 * c - 2), w1 = lds32(at + 8 * c + 2), w2 = lds32(at + 8 * c + 6);
                        w[r][0] = __funnelshift_r(w0, w1, 16);
                        w[r][1] = __funnelshift_r(w1, w2, 16);
                    }
                } else {
                    const uint32_t q = RAG ? RowA2(at + 4 * c).word(0) : b & 1 ? lds32(at + 4 * c)
                                           : __funnelshift_r(lds32(at + 4 * c - 2), lds32(at + 4 * c + 2), 16);
                    if constexpr (TY == T_Q4_0) {  // q - 8 as signed bytes, without a carry between them
                        w[r][0] = (((q & ml) | 0x80808080u) - 0x08080808u) ^ 0x80808080u;
                        w[r][1] = (((q >> 4 & ml) | 0x80808080u) - 0x08080808u) ^ 0x80808080u;
                    } else {
                        const uint2 v = iq4nl_word(q);
                        w[r][0] = v.x;
                        w[r][1] = v.y;
                    }
                }
            }
            int d[NS][4];
            X.template mma<true>(d, b, w[0][0], w[1][0], w[0][1], w[1][1]);
            float v[NV][2];
            wide_join<MODE, true>(d, v);
            float da = f16bits(lds16(ua + BB * b)), db = f16bits(lds16(ub + BB * b));
            if (RAG && (uint32_t)b >= left) da = db = 0.f;
#pragma unroll
            for (int i = 0; i < NV; i++) {
                sum[i][0] = fmaf(da, v[i][0], sum[i][0]);
                sum[i][1] = fmaf(db, v[i][1], sum[i][1]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < NV; i++) {
        acc[i][0] = fmaf(X.scale[i], sum[i][0], acc[i][0]);
        acc[i][1] = fmaf(X.scale[i], sum[i][1], acc[i][1]);
    }
}

}  // namespace okf
