// Prefill matmul on the 5th-generation tensor cores: out[n][m] = sum_k X[n][k] W[m][k]
// for N >= 9 tokens; the kernel for more than 256 tokens (and for fp32 activations that nobody could convert), the
// plans for it and for the one of okf_gemm_ts.cu, and the reduction of both.  Replaces the reference's gemm_mm_impl tile
// (LLM/metal/Kernels.metal:226-294), which stages fp16 copies of a 64 x 32
// weight tile and a 32 x 32 activation tile for simdgroup matrices.
//
// Shape of the computation.  One work item is a 128-row slab of W against two
// blocks of 256 tokens at once, so that every unpacked weight
// tile feeds two accumulators (fp32 activations: one block).  Per k-block of 64:
//   - the activation tile(s), 256 tokens x 64 k each, come by TMA through a tensor
//     map of X, already in the 128-byte-swizzled K-major layout the tensor core
//     reads (fp32 activations are converted to bf16 once per call before; where there is no memory for
//     that, eight warps convert them tile by tile and the other eight unpack alone);
//   - two groups of eight warps, taking the k-blocks in turn, unpack 128 rows x 64
//     weights to 16-bit floats into the same layout; weight bytes are fetched one
//     or two turns ahead;
//   - one warp, converged, issues four tcgen05.mma (M = 128, N = 256, K = 16) per token block
//     that accumulate in fp32 in tensor memory: lane = weight row, column = token;
//   - tcgen05.commit hands the stage back to the producers when the MMAs that
//     read it are done.
// The two 256-column accumulators of tensor memory serve the two token
// blocks of an item (fp32 activations: alternate between items).  What bounds it: power in long runs, else the tensor core's
// issue.  (Tried: pairs of CTAs with cta_group::2 on 256 rows x 512 tokens, half the activations' traffic: Q4_K 5120 -> 17408, 512
// tokens, 76.7 us against 69.1, 4096 tokens 599 against 565; 71 and 551 with no unpacking at all.)  Operands are
// fp16 when the activations are fp16, bf16 otherwise (fp32 activations are
// rounded to bf16); weights are decoded in fp32, exactly but for the mins of Q4_K and Q5_K (below), and
// rounded once.
//
// Every mbarrier wait is bounded (about a second); a wait that gives up records
// a code in the status word, the CTA frees its tensor memory and returns.
#include <cstring>

#include "okf_tc.cuh"
#include "okf_gemm_ts.h"
#include "okf_gemv_wide.cuh"
#include "okf_internal.h"
#include "okf_kernels.h"

namespace okf {

namespace tc {

constexpr uint32_t kABytes = kBM * kBK * 2;  // 16 KB
constexpr uint32_t kBBytes = kBN * kBK * 2;  // 32 KB per 256 tokens
// Two rings.  With one token block per item (fp32 activations) four stages of A (16 KB) and of B (32 KB).  With
// two blocks a B stage is 64 KB: three of them and two of A, so that a B tile has two MMA
// periods to arrive while the next A tile only has to be stored (IQ2_XXS, which also keeps its
// codebook in shared memory, stays with two B stages).
constexpr uint32_t kAWarps = 8;                        // warps 0..7 unpack weights (A tile)
constexpr uint32_t kBWarps = 8;                        // warps 8..15: fp32 activations: convert the B tile;
                                                       // 16-bit activations: a second unpacking group
constexpr uint32_t kProducerWarps = kAWarps + kBWarps;
constexpr uint32_t kTmaWarp = kProducerWarps;          // warp 16: hands B tiles to the copy engine
constexpr uint32_t kMmaWarp = kProducerWarps + 1;      // warp 17
constexpr uint32_t kThreads = (kProducerWarps + 2 + 4) * 32;  // + four epilogue warps
constexpr uint32_t kMaxRing = 4;                                      // stages the rings may have
constexpr uint32_t kBarRegion = 512;                                  // barriers, tensor-memory slot, abort flag
template <int TY, int NACC> struct Rings {
    static constexpr uint32_t a_stages = NACC == 2 ? 2 : 4;
    static constexpr uint32_t b_stages = NACC == 2 ? (TY == T_IQ2_XXS ? 2 : 3) : 4;
    static constexpr uint32_t a_bytes = a_stages * kABytes, b_stage = NACC * kBBytes, b_bytes = b_stages * b_stage;
    static constexpr uint32_t grid_bytes = TY == T_IQ2_XXS ? 2048 : 0;
    static constexpr uint32_t smem = 1024 /*align*/ + a_bytes + b_bytes + grid_bytes + kBarRegion;
};
struct Args {
    const uint8_t *w;
    const void *x;
    void *out;
    int *status;
    uint32_t k, m, n;
    uint32_t row_bytes;
    uint32_t waves;    // whole items every CTA takes before the dealt ones
    uint32_t dealt;    // items whose k-blocks are dealt out evenly (0: all items are whole) ...
    uint32_t dealers;  // ... over this many of the CTAs; every one of them gets some
    uint32_t nt;       // tokens of a partial tile
    float *partial;    // dealt items: fp32 partial tiles [part][dealt item][nt][128], summed by a second kernel
};
// Row shards: where results go instead of Args::out.  `nout` buffers (every rank's copy of
// the whole output as mapped here), element (token, row) at [token * out_ld + out_row0 + row].
// A parameter of its own: the main loops compile to slower code (fewer registers, 12 % less
// throughput measured) when Args grows.
struct Outs {
    uint32_t nout, out_ld, out_row0;
    void *outs[8];
    uint32_t *epoch;      // the local count the exchange is complete at goes up by epoch_inc
    uint32_t epoch_inc;
};

// One piece of work of a CTA: rows [mt * 128, +128) x tokens [n0, n0 + ntok) x k-blocks [kb0, kb1).
struct Work {
    uint32_t mt, n0, ntok, kb0, kb1;
    uint32_t slot;  // which partial tile it is: part * dealt + item; kWhole: it is all of K and goes to the output
};
constexpr uint32_t kWhole = 0xFFFFFFFFu;

// The j-th piece of work of this CTA; false when there is none.  Whole items go
// round-robin over the CTAs, then every CTA takes its run of the dealt k-blocks, item after item.
template <int NACC>
__device__ __forceinline__ bool next_work(const Args &p, uint32_t j, Work &w) {
    const uint32_t n_groups = (p.n + NACC * kBN - 1) / (NACC * kBN);
    const uint32_t base = ((p.m + kBM - 1) / kBM) * n_groups, kblocks = p.k / kBK;
    uint32_t item;
    w.ntok = NACC * kBN;
    w.slot = kWhole;
    w.kb0 = 0;
    w.kb1 = kblocks;
    if (!p.dealt || j < p.waves) {
        item = blockIdx.x + j * gridDim.x;
        if (item >= base) return false;
    } else {
        const uint32_t total = p.dealt * kblocks;
        if (blockIdx.x >= p.dealers) return false;
        const uint32_t lo = total * blockIdx.x / p.dealers, hi = total * (blockIdx.x + 1) / p.dealers;
        const uint32_t i = lo / kblocks + (j - p.waves), start = max(lo, i * kblocks), end = min(hi, (i + 1) * kblocks);
        if (start >= end) return false;
        w.kb0 = start - i * kblocks;
        w.kb1 = end - i * kblocks;
        if (w.kb1 - w.kb0 < kblocks) w.slot = (blockIdx.x - dealt_to(i * kblocks, total, p.dealers)) * p.dealt + i;
        item = base - p.dealt + i;
    }
    w.mt = item / n_groups;
    w.n0 = (item % n_groups) * (NACC * kBN);
    return true;
}

// ---- weights for the A tile -------------------------------------------------------
// ARaw<TY> holds, in registers, the bytes one thread needs to unpack 32 weights (half h of k-block kb) of
// its row; load() is issued a turn or two ahead of unpack() so that the latency of L2 hides behind the
// work in between.  unpack() leaves four groups of eight 16-bit floats; chunk() says which 16-byte chunk
// of the row's 128 bytes (64 k) each group is.
//
// A code byte becomes a float by one byte permute that puts it into the mantissa of a constant: 128 + b
// for codes below 128 (mantissa bits 16 .. 22), 32768 + b for whole bytes (bits 8 .. 15).  The constant's
// share leaves through the addend of the multiply-add that applies the scale, scale * (X + b) + add: one
// permute, one FMA and half a conversion per weight.  The addend is exact for every type without mins
// (a scale has 11 to 18 significant bits, the constants 3 to 9), so weights are still decoded exactly and
// rounded once; with mins it is off by 2^-24 of 128 scales, 1 / 500 of the rounding to fp16.
// (Before, the types other than Q4_K, Q8_0 and Q2_0 were unpacked byte by byte from memory: Q5_K 5120 ->
// 17408 at 64 tokens took 224 us, so 53; with the 8-byte loads below 5120 -> 18944 takes Q6_K 59, IQ4_NL 44.)
__device__ __forceinline__ float code_f32(uint32_t word, int byte) { return __uint_as_float(__byte_perm(word, 0x43000000u, 0x7044 | byte << 8)); }
__device__ __forceinline__ float wide_f32(uint32_t word, int byte) { return __uint_as_float(__byte_perm(word, 0x47000000u, 0x7404 | byte << 4)); }
// four weights out of the bytes of a word
template <bool F16>
__device__ __forceinline__ uint2 unpack4(uint32_t w, float mul, float add) {
    return make_uint2(pack16<F16>(fmaf(mul, code_f32(w, 0), add), fmaf(mul, code_f32(w, 1), add)),
                      pack16<F16>(fmaf(mul, code_f32(w, 2), add), fmaf(mul, code_f32(w, 3), add)));
}
template <bool F16>
__device__ __forceinline__ uint4 unpack8(uint32_t w0, uint32_t w1, float mul, float add) {
    const uint2 a = unpack4<F16>(w0, mul, add), b = unpack4<F16>(w1, mul, add);
    return make_uint4(a.x, a.y, b.x, b.y);
}
// 4 * NW bytes at a 2-byte aligned global address: aligned words (the last may lie past the block:
// buffers are padded) and, in get(), a funnel shift
template <int NW> struct Ldg2 {
    uint32_t w[NW + 1], sh;
    __device__ __forceinline__ void load(const uint8_t *b) {
        const uint32_t *p = reinterpret_cast<const uint32_t *>(reinterpret_cast<uintptr_t>(b) & ~(uintptr_t)3);
        sh = ((uint32_t)reinterpret_cast<uintptr_t>(b) & 2u) * 8u;
#pragma unroll
        for (int i = 0; i <= NW; i++) w[i] = __ldg(p + i);
    }
    __device__ __forceinline__ uint32_t get(int i) const { return __funnelshift_r(w[i], w[i + 1], sh); }
};
// The same from the NL aligned 8-byte words that hold it: sixteen rows a warp apart, every load costs the
// L1 sixteen look-ups however wide it is, and the types with 2-byte aligned blocks were bound by them (5120 ->
// 18944, 64 tokens, with 4-byte words: Q8_0 67 -> 46 us, Q6_K 64 -> 59, Q4_0 44 -> 37, IQ4_NL 47 -> 44).
template <int NW, int NL> struct Ldg8 {
    uint2 v[NL];
    uint32_t off;  // the bytes' place in the first word: 0, 2, 4 or 6
    __device__ __forceinline__ void load(const uint8_t *b) {
        const uint2 *p = reinterpret_cast<const uint2 *>(reinterpret_cast<uintptr_t>(b) & ~(uintptr_t)7);
        off = (uint32_t)reinterpret_cast<uintptr_t>(b) & 6u;
#pragma unroll
        for (int i = 0; i < NL; i++) v[i] = __ldg(p + i);
    }
    __device__ __forceinline__ uint32_t word(int i) const {
        i = i < 2 * NL ? i : 2 * NL - 1;  // past the bytes that count
        return i & 1 ? v[i >> 1].y : v[i >> 1].x;
    }
    __device__ __forceinline__ uint32_t half(int i) const { return off & 4u ? word(i + 1) : word(i); }
    __device__ __forceinline__ uint32_t get(int i) const { return __funnelshift_r(half(i), half(i + 1), (off & 2u) * 8u); }
};
__device__ __forceinline__ uint32_t chunk_in_order(uint32_t h, uint32_t c4) { return h * 4 + c4; }

template <int TY> struct ARaw;
// Q4_K, Q5_K: a k-block is 32 bytes of qs: low nibbles = its first 32 weights (sub-block 2p), high
// nibbles = the other 32 (sub-block 2p + 1); Q5_K's fifth bit of sub-block j is bit j of qh[l].  The two
// threads of a row take 16 bytes each and unpack both nibbles: 32 bytes of Q4_K per k-block and thread,
// header included, and two k-blocks in flight: one turn ahead does not cover the latency of L2.
template <int TY> struct ARawK45 {
    static constexpr int kAhead = 2;  // k-blocks of this thread in flight beside the one being unpacked
    // values 0..15 are k = 16h + 0..15 (chunks 2h, 2h + 1), values 16..31 the same positions 32 further on
    __device__ static __forceinline__ uint32_t chunk(uint32_t h, uint32_t c4) { return (c4 >> 1) * 4 + 2 * h + (c4 & 1); }
    uint4 hdr, q, h5;
    uint32_t p;  // which 32 bytes of the block's 128
    __device__ __forceinline__ void load(const uint8_t *row, uint32_t kb, uint32_t h) {
        const uint8_t *b = row + (size_t)(kb >> 2) * (TY == T_Q4_K ? 144 : 176);
        p = kb & 3;
        if constexpr (TY == T_Q4_K) {  // 16-byte aligned
            hdr = __ldg(reinterpret_cast<const uint4 *>(b));
            q = __ldg(reinterpret_cast<const uint4 *>(b + 16 + 32 * p + 16 * h));
        } else if (((uintptr_t)b & 15) == 0) {
            hdr = __ldg(reinterpret_cast<const uint4 *>(b));
            h5 = __ldg(reinterpret_cast<const uint4 *>(b + 16 + 16 * h));
            q = __ldg(reinterpret_cast<const uint4 *>(b + 48 + 32 * p + 16 * h));
        } else {  // a tensor that does not start on a 16-byte boundary
            auto ld = [](const uint8_t *a) { return make_uint4(ld_u32_a2(a), ld_u32_a2(a + 4), ld_u32_a2(a + 8), ld_u32_a2(a + 12)); };
            hdr = ld(b);
            h5 = ld(b + 16 + 16 * h);
            q = ld(b + 48 + 32 * p + 16 * h);
        }
    }
    // w = (d * sc) * q - dmin * m (LLM/Quantize/KQuants.swift:104-158)
    template <bool F16> __device__ __forceinline__ void unpack(uint4 (&o)[4], const uint32_t *) const {
        // 6-bit scales and mins of sub-blocks 2p and 2p + 1 (get_scale_min_k4): bytes 2p, 2p + 1 of
        // the scale field for p < 2, split fields above
        const uint32_t sh = (p & 1) * 16;
        const uint32_t a = hdr.y >> sh, b = hdr.z >> sh, e = hdr.w >> sh;
        uint32_t sc, mn;  // two bytes each: sub-block 2p, 2p + 1
        if (p < 2) { sc = a & 0x3F3Fu; mn = b & 0x3F3Fu; }
        else { sc = (e & 0x0F0Fu) | ((a >> 2) & 0x3030u); mn = ((e >> 4) & 0x0F0Fu) | ((b >> 2) & 0x3030u); }
        const float d = f16bits(hdr.x & 0xFFFF), dm = f16bits(hdr.x >> 16);
        const float d0 = d * byte_to_f32(sc, 0), d1 = d * byte_to_f32(sc, 1);
        const float o0 = fmaf(d0, -128.f, -dm * byte_to_f32(mn, 0)), o1 = fmaf(d1, -128.f, -dm * byte_to_f32(mn, 1));
        const uint32_t w[4] = {q.x, q.y, q.z, q.w}, f[4] = {h5.x, h5.y, h5.z, h5.w};
        uint32_t lo[4], hi[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            lo[i] = w[i] & 0x0F0F0F0Fu;
            hi[i] = (w[i] >> 4) & 0x0F0F0F0Fu;
            if constexpr (TY == T_Q5_K) {
                const uint32_t t = f[i] >> (2 * p);
                lo[i] |= (t << 4) & 0x10101010u;
                hi[i] |= (t << 3) & 0x10101010u;
            }
        }
        o[0] = unpack8<F16>(lo[0], lo[1], d0, o0);
        o[1] = unpack8<F16>(lo[2], lo[3], d0, o0);
        o[2] = unpack8<F16>(hi[0], hi[1], d1, o1);
        o[3] = unpack8<F16>(hi[2], hi[3], d1, o1);
    }
};
template <> struct ARaw<T_Q4_K> : ARawK45<T_Q4_K> {};
template <> struct ARaw<T_Q5_K> : ARawK45<T_Q5_K> {};
// Q6_K: k-block kb is granules r = 2 (kb & 1), + 1 of half n of the block: 64 bytes of ql (low nibbles for
// even kb, high for odd) and 32 of qh.  The two threads of a row take positions 16h .. 16h + 15 of both
// granules, one scale each.
template <> struct ARaw<T_Q6_K> {
    static constexpr int kAhead = 1;
    __device__ static __forceinline__ uint32_t chunk(uint32_t h, uint32_t c4) { return (c4 >> 1) * 4 + 2 * h + (c4 & 1); }
    Ldg8<4, 3> l0, l1, hq;
    uint32_t sc, par;
    float d;
    __device__ __forceinline__ void load(const uint8_t *row, uint32_t kb, uint32_t h) {
        const uint8_t *b = row + (size_t)(kb >> 2) * 210;
        const uint32_t n = (kb >> 1) & 1;
        par = kb & 1;
        l0.load(b + 64 * n + 16 * h);
        l1.load(b + 64 * n + 32 + 16 * h);
        hq.load(b + 128 + 32 * n + 16 * h);
        const uint8_t *s = b + 192 + 8 * n + 4 * par + h;
        sc = (uint32_t)__ldg(s) | (uint32_t)__ldg(s + 2) << 8;
        d = f16bits(__ldg(reinterpret_cast<const uint16_t *>(b + 208)));
    }
    // d * scale * (q - 32) (LLM/Quantize/KQuants.swift:160-177)
    template <bool F16> __device__ __forceinline__ void unpack(uint4 (&o)[4], const uint32_t *) const {
        const float m0 = d * (float)(int)(int8_t)(sc & 0xFF), m1 = d * (float)(int)(int8_t)(sc >> 8 & 0xFF);
        uint32_t a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint32_t h = hq.get(i) >> (4 * par);
            a[i] = ((l0.get(i) >> (4 * par)) & 0x0F0F0F0Fu) | ((h << 4) & 0x30303030u);
            b[i] = ((l1.get(i) >> (4 * par)) & 0x0F0F0F0Fu) | ((h << 2) & 0x30303030u);
        }
        o[0] = unpack8<F16>(a[0], a[1], m0, -160.f * m0);
        o[1] = unpack8<F16>(a[2], a[3], m0, -160.f * m0);
        o[2] = unpack8<F16>(b[0], b[1], m1, -160.f * m1);
        o[3] = unpack8<F16>(b[2], b[3], m1, -160.f * m1);
    }
};
template <> struct ARaw<T_Q8_0> {
    static constexpr int kAhead = 1;
    __device__ static __forceinline__ uint32_t chunk(uint32_t h, uint32_t c4) { return chunk_in_order(h, c4); }
    Ldg8<9, 5> w;  // the 34-byte block {f16 d; i8 q[32]}
    __device__ __forceinline__ void load(const uint8_t *row, uint32_t kb, uint32_t h) { w.load(row + (size_t)(kb * 2 + h) * 34); }
    template <bool F16> __device__ __forceinline__ void unpack(uint4 (&o)[4], const uint32_t *) const {
        uint32_t u[9];
#pragma unroll
        for (int i = 0; i < 9; i++) u[i] = w.get(i) ^ (i ? 0x80808080u : 0x80800000u);  // q + 128 as unsigned bytes
        const float d = f16bits(u[0] & 0xFFFF), add = -32896.f * d;
        auto val = [&](int j) { return fmaf(d, wide_f32(u[(j + 2) >> 2], (j + 2) & 3), add); };
#pragma unroll
        for (int c = 0; c < 4; c++)
            o[c] = make_uint4(pack16<F16>(val(8 * c), val(8 * c + 1)), pack16<F16>(val(8 * c + 2), val(8 * c + 3)),
                              pack16<F16>(val(8 * c + 4), val(8 * c + 5)), pack16<F16>(val(8 * c + 6), val(8 * c + 7)));
    }
};
// Q4_0, IQ4_NL: {f16 d; u8 qs[16]}, byte j = weights j (low nibble) and j + 16 (high)
template <int TY> struct ARaw40 {
    static constexpr int kAhead = 1;
    __device__ static __forceinline__ uint32_t chunk(uint32_t h, uint32_t c4) { return chunk_in_order(h, c4); }
    Ldg8<5, 3> w;
    __device__ __forceinline__ void load(const uint8_t *row, uint32_t kb, uint32_t h) { w.load(row + (size_t)(kb * 2 + h) * 18); }
    template <bool F16> __device__ __forceinline__ void unpack(uint4 (&o)[4], const uint32_t *) const {
        uint32_t u[5], q[4];
#pragma unroll
        for (int i = 0; i < 5; i++) u[i] = w.get(i);
        const float d = f16bits(u[0] & 0xFFFF);
#pragma unroll
        for (int i = 0; i < 4; i++) q[i] = __funnelshift_r(u[i], u[i + 1], 16);
        if constexpr (TY == T_Q4_0) {
            const float add = -136.f * d;
            constexpr uint32_t ml = 0x0F0F0F0Fu;
            o[0] = unpack8<F16>(q[0] & ml, q[1] & ml, d, add);
            o[1] = unpack8<F16>(q[2] & ml, q[3] & ml, d, add);
            o[2] = unpack8<F16>(q[0] >> 4 & ml, q[1] >> 4 & ml, d, add);
            o[3] = unpack8<F16>(q[2] >> 4 & ml, q[3] >> 4 & ml, d, add);
        } else {
            // the codebook's values + 128 (LLM/Gemma/Gemma4Quant.swift:5-9), looked up eight nibbles a word in the
            // order they follow: lo, hi of byte 0, lo, hi of byte 1, ... (see iq4nl_word)
            constexpr uint32_t T0 = 0x3F2D1801u, T1 = 0x766A5D4Fu, T2 = 0xA6998D81u, T3 = 0xF1D9C5B5u;
            const float add = -32896.f * d;
            uint32_t t[8];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t sel = q[i] & 0x77777777u, pick = (q[i] >> 1 & 0x44444444u) | 0x32103210u;
                t[2 * i] = __byte_perm(__byte_perm(T0, T1, sel), __byte_perm(T2, T3, sel), pick);
                t[2 * i + 1] = __byte_perm(__byte_perm(T0, T1, sel >> 16), __byte_perm(T2, T3, sel >> 16), pick >> 16);
            }
            auto val = [&](int j) { return fmaf(d, wide_f32(t[(j & 15) >> 1], (j & 1) * 2 + (j >> 4)), add); };
#pragma unroll
            for (int c = 0; c < 4; c++)
                o[c] = make_uint4(pack16<F16>(val(8 * c), val(8 * c + 1)), pack16<F16>(val(8 * c + 2), val(8 * c + 3)),
                                  pack16<F16>(val(8 * c + 4), val(8 * c + 5)), pack16<F16>(val(8 * c + 6), val(8 * c + 7)));
        }
    }
};
template <> struct ARaw<T_Q4_0> : ARaw40<T_Q4_0> {};
template <> struct ARaw<T_IQ4_NL> : ARaw40<T_IQ4_NL> {};
template <> struct ARaw<T_Q2_0> {
    static constexpr int kAhead = 2;
    __device__ static __forceinline__ uint32_t chunk(uint32_t h, uint32_t c4) { return chunk_in_order(h, c4); }
    Ldg2<2> w;  // 32 two-bit codes
    uint32_t dbits;
    __device__ __forceinline__ void load(const uint8_t *row, uint32_t kb, uint32_t h) {
        const uint8_t *b = row + (size_t)(kb >> 1) * 34;  // block of 128 weights
        dbits = __ldg(reinterpret_cast<const uint16_t *>(b));
        w.load(b + 2 + 16 * (kb & 1) + 8 * h);
    }
    template <bool F16> __device__ __forceinline__ void unpack(uint4 (&o)[4], const uint32_t *) const {
        const float d = f16bits(dbits), add = -129.f * d;  // (code - 1) * d
        uint32_t t[2][4];
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int e = 0; e < 4; e++) t[i][e] = w.get(i) >> (2 * e) & 0x03030303u;  // byte b: code 4b + e
        auto val = [&](int j) { return fmaf(d, code_f32(t[j >> 4][j & 3], (j & 15) >> 2), add); };
#pragma unroll
        for (int c = 0; c < 4; c++)
            o[c] = make_uint4(pack16<F16>(val(8 * c), val(8 * c + 1)), pack16<F16>(val(8 * c + 2), val(8 * c + 3)),
                              pack16<F16>(val(8 * c + 4), val(8 * c + 5)), pack16<F16>(val(8 * c + 6), val(8 * c + 7)));
    }
};
// IQ2_XXS: sub-block = {u32: four codebook indices, u32: four 7-bit sign indices + 4-bit scale}
// (LLM/Quantize/IQ2XXS.swift:34-53).  The tables in shared memory hold byte-permute selectors (see
// iq2_code_selectors): over the magnitudes and their negatives, all 64 up so that they are below 128.
template <> struct ARaw<T_IQ2_XXS> {
    static constexpr int kAhead = 2;
    __device__ static __forceinline__ uint32_t chunk(uint32_t h, uint32_t c4) { return chunk_in_order(h, c4); }
    Ldg2<2> w;
    uint32_t dbits;
    __device__ __forceinline__ void load(const uint8_t *row, uint32_t kb, uint32_t h) {
        const uint8_t *b = row + (size_t)(kb >> 2) * 66;
        dbits = __ldg(reinterpret_cast<const uint16_t *>(b));
        w.load(b + 2 + 8 * ((kb & 3) * 2 + h));
    }
    template <bool F16> __device__ __forceinline__ void unpack(uint4 (&o)[4], const uint32_t *tab) const {
        const uint32_t a0 = w.get(0), a1 = w.get(1);
        const float db = f16bits(dbits) * (0.5f + (float)(a1 >> 28)) * 0.25f, add = -192.f * db;
        constexpr uint32_t P = 0x406B5948u, N = 0x40152738u;  // 64 + {8, 25, 43, 0}, 64 - {8, 25, 43, 0}
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const uint32_t s = tab[__byte_perm(a0, 0u, 0x4440 + c)] | tab[256 + (a1 >> (7 * c) & 127u)];
            o[c] = unpack8<F16>(__byte_perm(P, N, s), __byte_perm(P, N, s >> 16), db, add);
        }
    }
};

// NACC: token blocks (accumulators) per work item, 1 or 2.
template <int TY, int XDT, typename OT, int NACC>
// (The tensor map comes first so that its 128 bytes start on a 128-byte boundary of the
// parameter block whatever the size of Args: measured 12 % slower when it straddled one.)
__global__ void __launch_bounds__(kThreads, 1) gemm_tc_kernel(const __grid_constant__ CUtensorMap xmap, Args p, Outs go) {
    constexpr bool F16 = XDT == DT_F16;
    constexpr bool ASYNC_B = XDT != DT_F32;  // 16-bit activations come by TMA, fp32 ones are converted by eight warps
    using R = Rings<TY, NACC>;
    constexpr uint32_t kAStages = Rings<TY, NACC>::a_stages, kBStages = Rings<TY, NACC>::b_stages, kBStage = Rings<TY, NACC>::b_stage;
    constexpr uint32_t kGroups = ASYNC_B ? 2 : 1;  // groups of eight unpacking warps
    static_assert(kAStages % kGroups == 0, "a stage belongs to one group, which so waits for every phase of its barriers");
    static_assert(kAStages <= kMaxRing && kBStages <= kMaxRing, "room for the barriers");
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t *a_ring = smem, *b_ring = smem + kAStages * kABytes;
    uint32_t *tab = reinterpret_cast<uint32_t *>(smem + R::a_bytes + R::b_bytes);  // IQ2_XXS: 256 + 128 selector words
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + R::a_bytes + R::b_bytes + R::grid_bytes);
    uint64_t *full_a = bars, *empty_a = bars + kMaxRing;                    // A producers <-> MMA, one pair per A stage
    uint64_t *full_b = bars + 2 * kMaxRing, *empty_b = full_b + kMaxRing;  // B producer(s) <-> MMA, one pair per B stage
    uint64_t *acc_full = empty_b + kMaxRing;  // MMA -> epilogue, one per accumulator
    uint64_t *acc_empty = acc_full + 2;        // epilogue -> MMA
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_full + 4);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

    const uint32_t warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;  // (uniform, and known to be)
    pdl_launch_dependents();
    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < kAStages; s++) {
            mbar_init(&full_a[s], kAWarps);
            mbar_init(&empty_a[s], 1);
        }
        for (uint32_t s = 0; s < kBStages; s++) {
            mbar_init(&full_b[s], ASYNC_B ? 1 : kBWarps);
            mbar_init(&empty_b[s], 1);
        }
        for (uint32_t a = 0; a < 2; a++) {
            mbar_init(&acc_full[a], 1);
            mbar_init(&acc_empty[a], 4);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if constexpr (TY == T_IQ2_XXS) {
        for (uint32_t i = threadIdx.x; i < 384; i += kThreads) tab[i] = i < 256 ? iq2_code_selectors(g_iq2xxs_grid[i]) : iq2_sign_selectors(i - 256);
    }
    if (warp == kMmaWarp) {
        // the whole tensor memory of the SM: two 256-column accumulators
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp < kAWarps || (ASYNC_B && warp < kProducerWarps)) {
        // ---------------- A producers: unpack 128 rows x 64 weights into swizzled shared memory.
        // With 16-bit activations there are two groups of eight warps that take the k-blocks
        // in turn: one k-block's latency (load, decode, wait, store, fence) is longer than the
        // MMAs it feeds, two in flight are not.
        const uint32_t grp = warp / kAWarps;
        const uint32_t t = threadIdx.x % (kAWarps * 32);
        // Thread t unpacks 32 weights of row arow.  Eight lanes in a row have eight rows and the same half, so that their 16-byte
        // stores fall on eight bank groups (two halves of four rows: two lanes to a group for the types with super-blocks, 128
        // cycles of a k-block's 1500 at the shared-memory port).
        const uint32_t arow = (t >> 4) * 8 + (t & 7), ahalf = t >> 3 & 1;
        uint32_t it0 = 0;  // stage counter at the start of the work item
        Work wk;
        // this thread's four 16-byte chunks -> stage s
        // (a group's stages follow each other across work items: every kGroups-th of the ring)
        uint32_t s = grp, use = 0;
        auto put = [&](const uint4 (&q)[4]) -> bool {
            if (use > 0 && !warp_wait(&empty_a[s], (use - 1) & 1, lane, abort_flag, p.status)) return false;
            const uint32_t sa = smem_u32(a_ring) + s * kABytes;
#pragma unroll
            for (int c4 = 0; c4 < 4; c4++)
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(sa + swz(arow, ARaw<TY>::chunk(ahalf, c4))), "r"(q[c4].x),
                             "r"(q[c4].y), "r"(q[c4].z), "r"(q[c4].w)
                             : "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&full_a[s]);  // the MMA issuer fences these stores for the tensor core
            s += kGroups;
            if (s >= kAStages) {
                s -= kAStages;
                use++;
            }
            return true;
        };
        for (uint32_t j = 0; next_work<NACC>(p, j, wk); j++) {
            const uint32_t m0 = wk.mt * kBM;
            const uint32_t kb0 = wk.kb0, kb1 = wk.kb1;
            const uint32_t wrow = min(m0 + arow, p.m - 1);  // rows past the end repeat the last one; nobody stores them
            const uint8_t *wp = p.w + (size_t)wrow * p.row_bytes;
            // this group's first k-block: the one whose stage counter has its parity
            const uint32_t first = kb0 + (kGroups == 2 ? ((grp + it0) & 1) : 0);
            // The bytes of the next k-block (Q4_K: of the next two) are fetched while this one is
            // unpacked.  (Tried and slower: refilling a register set only after put(), whose proxy
            // fence waits for the loads in flight; three sets taking turns without moves.)
            if constexpr (ARaw<TY>::kAhead == 2) {
                ARaw<TY> cur, n1, n2;
                if (first < kb1) cur.load(wp, first, ahalf);
                if (first + kGroups < kb1) n1.load(wp, first + kGroups, ahalf);
                for (uint32_t kb = first; kb < kb1; kb += kGroups) {
                    if (kb + 2 * kGroups < kb1) n2.load(wp, kb + 2 * kGroups, ahalf);
                    uint4 v[4];
                    cur.template unpack<F16>(v, tab);
                    if (!put(v)) goto done;
                    cur = n1;
                    n1 = n2;
                }
            } else {
                ARaw<TY> cur, nxt;
                if (first < kb1) cur.load(wp, first, ahalf);
                for (uint32_t kb = first; kb < kb1; kb += kGroups) {
                    if (kb + kGroups < kb1) nxt.load(wp, kb + kGroups, ahalf);  // lands while cur is unpacked
                    uint4 v[4];
                    cur.template unpack<F16>(v, tab);
                    if (!put(v)) goto done;
                    cur = nxt;
                }
            }
            it0 += kb1 - kb0;
        }
    } else if (warp == kTmaWarp) {
        // ---------------- hands the B tiles of 16-bit activations to the copy engine: NACC x 256 tokens x 64 k a stage
        if constexpr (ASYNC_B) {
            pdl_wait();  // x may come from the kernel before
            uint32_t s = 0, use = 0;
            Work wk;
            for (uint32_t j = 0; next_work<NACC>(p, j, wk); j++) {
                const uint32_t nblk = wk.ntok > kBN ? NACC : 1;
                for (uint32_t kb = wk.kb0; kb < wk.kb1; kb++, s = s + 1 == kBStages ? (use++, 0) : s + 1) {
                    if (use > 0 && !warp_poll(&empty_b[s], (use - 1) & 1, abort_flag, p.status)) {
                        // giving up: the copies already handed over land within microseconds;
                        // stay for a while so that they do not write into a CTA that has gone
                        const long long t0 = clock64();
                        while (clock64() - t0 < 100000) {}
                        goto done;
                    }
                    uint8_t *sb = b_ring + (size_t)s * kBStage;
                    if (elect_one()) {
                        mbar_expect_tx(&full_b[s], nblk * kBBytes);
                        for (uint32_t a = 0; a < nblk; a++)
                            tma_load_tile(sb + a * kBBytes, &xmap, kb * kBK, wk.n0 + a * kBN, &full_b[s]);
                    }
                    __syncwarp();
                }
            }
        }
    } else if (warp < kProducerWarps) {
        // ---------------- B tiles of fp32 activations: eight warps convert them
        if constexpr (!ASYNC_B) {
            const uint32_t t = threadIdx.x - kAWarps * 32;  // 0..255
            constexpr uint32_t kChunks = NACC * kBN * 8 / (kBWarps * 32);  // 16-byte chunks per thread
            uint32_t s = 0, use = 0;
            Work wk;
            pdl_wait();
            const float *x = dep_ptr(reinterpret_cast<const float *>(p.x));
            for (uint32_t j = 0; next_work<NACC>(p, j, wk); j++) {
                const uint32_t n0 = wk.n0;
                for (uint32_t kb = wk.kb0; kb < wk.kb1; kb++, s = s + 1 == kBStages ? (use++, 0) : s + 1) {
                    if (use > 0 && !warp_wait(&empty_b[s], (use - 1) & 1, lane, abort_flag, p.status)) goto done;
                    uint8_t *sb = b_ring + (size_t)s * kBStage;
                    // only as many tokens as the MMA reads, in sixteens
                    const uint32_t rows = (min(min(wk.ntok, p.n - n0), NACC * kBN) + 15u) & ~15u;
#pragma unroll 4
                    for (uint32_t i = 0; i < kChunks; i++) {
                        const uint32_t q = t + kBWarps * 32 * i;
                        if ((q >> 3) >= rows) break;
                        const uint32_t row = q >> 3, c16 = q & 7;  // row over NACC x 256 tokens; blocks are 32 KB apart
                        const uint32_t tok = n0 + row;
                        uint8_t *dst = sb + (row >> 8) * kBBytes + swz(row & 255, c16);
                        const size_t e = (size_t)min(tok, p.n - 1) * p.k + (size_t)kb * kBK + c16 * 8;
                        uint4 v = make_uint4(0u, 0u, 0u, 0u);
                        if (tok < p.n && row < wk.ntok) {
                            const float4 f0 = ld_dep(reinterpret_cast<const float4 *>(x + e));
                            const float4 f1 = ld_dep(reinterpret_cast<const float4 *>(x + e) + 1);
                            v.x = pack16<false>(f0.x, f0.y); v.y = pack16<false>(f0.z, f0.w);
                            v.z = pack16<false>(f1.x, f1.y); v.w = pack16<false>(f1.z, f1.w);
                        }
                        *reinterpret_cast<uint4 *>(dst) = v;
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&full_b[s]);
                }
            }
        }
    } else if (warp == kMmaWarp) {
        // ---------------- MMA issuer
        uint32_t tile = 0, s_a = 0, use_a = 0, s_b = 0, use_b = 0;
        Work wk;
        for (uint32_t j = 0; next_work<NACC>(p, j, wk); j++, tile++) {
            // N of the instruction: the tokens each block of the item really has, in sixteens
            const uint32_t live = min(wk.ntok, p.n - wk.n0);
            uint32_t idesc[NACC];
#pragma unroll
            for (uint32_t a = 0; a < (uint32_t)NACC; a++) {
                const uint32_t nt = live > a * kBN ? min(live - a * kBN, kBN) : 0u;
                idesc[a] = instr_desc(F16 ? 0u : 1u, kBM, nt ? (nt + 15u) & ~15u : 16u);
            }
            // accumulators: both for a two-block item, alternating for one-block items
            const uint32_t acc0 = NACC == 2 ? 0 : (tile & 1), acc_use = NACC == 2 ? tile : (tile >> 1);
            if (acc_use > 0)
                for (uint32_t a = 0; a < (uint32_t)NACC; a++)
                    if (!warp_poll(&acc_empty[acc0 + a], (acc_use - 1) & 1, abort_flag, p.status)) goto done;
            tc_fence_after();
            const uint32_t kb0 = wk.kb0, kb1 = wk.kb1;
            for (uint32_t kb = kb0; kb < kb1; kb++, s_a = s_a + 1 == kAStages ? (use_a++, 0) : s_a + 1,
                          s_b = s_b + 1 == kBStages ? (use_b++, 0) : s_b + 1) {
                if (!warp_poll(&full_a[s_a], use_a & 1, abort_flag, p.status) ||
                    !warp_poll(&full_b[s_b], use_b & 1, abort_flag, p.status))
                    goto done;
                // Generic-proxy stores (unpacked weights) -> visible to the tensor core's async proxy: the
                // fence stands on the path from the stores over the barrier to the MMAs.  Here and not in
                // the storing threads, where it also waits for their loads in flight, a round trip to L2
                // or HBM on every turn.
                fence_proxy_async();
                tc_fence_after();
                const uint64_t da = smem_desc(smem_u32(a_ring) + s_a * kABytes);
                const uint64_t db = smem_desc(smem_u32(b_ring) + s_b * kBStage);
                if (elect_one()) {
#pragma unroll
                    for (uint32_t a = 0; a < (uint32_t)NACC; a++)
#pragma unroll
                        for (uint32_t k4 = 0; k4 < kBK / 16; k4++)
                            // 16 k = 32 bytes further along the swizzled 128-byte row
                            umma(tmem_base + (acc0 + a) * kBN, da + (uint64_t)(k4 * 2), db + (uint64_t)(a * (kBBytes >> 4) + k4 * 2), idesc[a],
                                 (kb != kb0 || k4 != 0) ? 1u : 0u);
                    umma_commit(&empty_a[s_a]);  // both stages are free once these MMAs have read them
                    umma_commit(&empty_b[s_b]);
                }
                __syncwarp();
            }
            if (elect_one())
                for (uint32_t a = 0; a < (uint32_t)NACC; a++) umma_commit(&acc_full[acc0 + a]);
            __syncwarp();
        }
    } else {
        // ---------------- epilogue: four warps, warp q reads tensor-memory lanes 32q .. 32q + 31
        const uint32_t q = warp & 3;  // a warp may only touch the lane quarter given by warp id % 4
        if (warp == kMmaWarp + 1 && lane == 0) {
            // nothing to do yet: asks L2 for the CTA's whole slabs of W (128 contiguous rows) ahead of the
            // producers, which then read them k-block by k-block, 32 bytes per row at a time.  (Asking only
            // for the k-range of dealt items, row by row, made short launches 2 us slower.)
            uint32_t last_mt = 0xFFFFFFFFu;
            Work wk;
            for (uint32_t j = 0; next_work<NACC>(p, j, wk); j++) {
                const uint32_t mt = wk.mt;
                if (mt == last_mt) continue;  // same slab as the previous item
                last_mt = mt;
                const uint32_t m0 = mt * kBM;
                const size_t bytes = (size_t)min(kBM, p.m - m0) * p.row_bytes;
                const uint8_t *base = p.w + (size_t)m0 * p.row_bytes;
                if (((uintptr_t)base & 15) == 0) {
                    for (size_t off = 0; off + 16 <= bytes; off += 32768) {
                        const uint32_t n = (uint32_t)min((size_t)32768, (bytes - off) & ~(size_t)15);
                        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(base + off), "r"(n) : "memory");
                    }
                }
            }
        }
        __syncwarp();
        uint32_t tile = 0;
        Work wk;
        pdl_wait();  // the kernel before may still read what is written here
        for (uint32_t j = 0; next_work<NACC>(p, j, wk); j++, tile++) {
            const uint32_t mt = wk.mt, n0 = wk.n0;
            const uint32_t n_end = min(p.n, n0 + wk.ntok);
            const uint32_t acc0 = NACC == 2 ? 0 : (tile & 1), acc_use = NACC == 2 ? tile : (tile >> 1);
            const uint32_t row = mt * kBM + q * 32 + lane;
            // partial tiles hold all 128 rows
            float *part = wk.slot != kWhole ? p.partial + (size_t)wk.slot * p.nt * kBM - (size_t)n0 * kBM + q * 32 + lane : nullptr;
            for (uint32_t a = 0; a < (uint32_t)NACC; a++) {
                const uint32_t acc = acc0 + a;
                if (!warp_wait(&acc_full[acc], acc_use & 1, lane, abort_flag, p.status)) goto done;
                tc_fence_after();
#pragma unroll 1
                for (uint32_t c0 = 0; c0 < kBN; c0 += 32) {
                    if (n0 + a * kBN + c0 >= n_end) break;  // nothing but padding from here on
                    uint32_t r[32];
                    tmem_ld32(tmem_base + ((q * 32) << 16) + acc * kBN + c0, r);
                    tmem_ld_wait();
                    if (part) {
#pragma unroll
                        for (int j = 0; j < 32; j++) {
                            const uint32_t tok = n0 + a * kBN + c0 + j;
                            if (tok < n_end) part[(size_t)tok * kBM] = __uint_as_float(r[j]);
                        }
                    } else if (row < p.m) {
                        if constexpr (!kIsGather<OT>) {
                            OT *out = reinterpret_cast<OT *>(p.out);
#pragma unroll
                            for (int j = 0; j < 32; j++) {
                                const uint32_t tok = n0 + a * kBN + c0 + j;
                                if (tok < n_end) {
                                    const float f = __uint_as_float(r[j]);
                                    if constexpr (sizeof(OT) == 4) out[(size_t)tok * p.m + row] = f;
                                    else out[(size_t)tok * p.m + row] = __float2bfloat16_rn(f);
                                }
                            }
                        } else {
                            // row shards: a warp stores 32 consecutive rows of one token (128 bytes) into
                            // every rank's buffer, over NVLink for the other ranks'
                            for (uint32_t o = 0; o < go.nout; o++) {
                                float *po = reinterpret_cast<float *>(go.outs[o]) + go.out_row0 + row;
#pragma unroll
                                for (int j = 0; j < 32; j++) {
                                    const uint32_t tok = n0 + a * kBN + c0 + j;
                                    if (tok < n_end) po[(size_t)tok * go.out_ld] = __uint_as_float(r[j]);
                                }
                            }
                        }
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[acc]);
            }
        }
    }
done:
    if constexpr (kIsGather<OT>)
        if (!p.dealt && blockIdx.x == 0 && threadIdx.x == 0) {
            pdl_wait();
            go.epoch[0] += go.epoch_inc;
        }
    tc_fence_before();
    __syncthreads();
    if (warp == kMmaWarp) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

// Sum the partial tiles of the dealt items, part after part (the order of k), into every output buffer:
// element (token, row) at [token * out_ld + out_row0 + row].  A block takes 16 tokens of an item, a warp
// the 128 rows of one token at a time.  (The parameters stay where they are: indexed by a variable, a by-value copy goes to
// local memory first, 32 stores a thread.)
struct ReduceOut {
    uint32_t nout, m, n, out_ld, out_row0;
    uint32_t dealt, base, steps, ctas, nt, groups, group_tok;  // the main kernel's dealing, an item being `steps` long
    void *outs[8];
    uint32_t *epoch;
    uint32_t epoch_inc;
};
constexpr uint32_t kReduceTok = 16;
// Shared memory that the reduction asks for and does not use: four CTAs to an SM.  They start on the SMs that the matmul leaves
// first, and without it eight of them gather there, as their 32 registers a thread allow.  (With 0 / 48 / 100 KB: IQ4_NL 6144 -> 1500, 40
// tokens, 13.3 / 12.7 / 11.7 us, Q5_K 9728 -> 2560, 77 tokens, 18.9 / 18.3 / 17.2, but 2560 -> 9728 16.3 / 16.1 / 16.9 and Q4_K 9728 ->
// 2560, 512 tokens, 29.9 / 30.5 / 31.9: with many blocks it is the SMs that run out.)
constexpr uint32_t kReduceSmem = 48 * 1024;
// VEC: fp32 results leave as 16-byte words, as every row of every output starts on a 16-byte boundary.  The host
// decides, from the addresses too: an fp32 output need only be 4-byte aligned (a view into a larger tensor).  Else the four
// neighbours of every thread are dealt out again, so that a warp stores 32 rows side by side.  (Stored as they are, 16 bytes
// apart, results in page-locked host memory cross PCIe in pieces: Q4_0 4096 -> 2071, 11 tokens, host to host 50.4 us, so 44.1.)
// (As a run-time flag: Q5_K 2560 -> 9728, 77 tokens, 21.4 us instead of 19.5.)
template <typename OT, bool VEC>
__global__ void __launch_bounds__(256) reduce_kernel(const float *part, const __grid_constant__ ReduceOut o) {
    pdl_launch_dependents();
    const uint32_t runs = (o.nt + kReduceTok - 1) / kReduceTok;
    const uint32_t i = blockIdx.x / runs, t0 = blockIdx.x % runs * kReduceTok, total = o.dealt * o.steps;
    const uint32_t c0 = dealt_to(i * o.steps, total, o.ctas), c1 = dealt_to((i + 1) * o.steps - 1, total, o.ctas);
    const uint32_t item = o.base - o.dealt + i, n0 = item % o.groups * o.group_tok;
    const uint32_t lane = threadIdx.x & 31, row0 = item / o.groups * kBM;
    pdl_wait();
    if (o.epoch && blockIdx.x == 0 && threadIdx.x == 0) o.epoch[0] += o.epoch_inc;
    if (c0 == c1) return;  // one CTA took the whole item and stored it
    const float *parts = dep_ptr(part);
    for (uint32_t t = t0 + (threadIdx.x >> 5); t < min(t0 + kReduceTok, o.nt); t += 8) {
        if (n0 + t >= o.n) break;
        // (partial tiles hold all 128 rows)
        const float *src = parts + ((size_t)i * o.nt + t) * kBM + 4 * lane;
        const size_t step = (size_t)o.dealt * o.nt * kBM;
        float4 v = ld_dep(reinterpret_cast<const float4 *>(src));
        for (uint32_t c = c0 + 1; c <= c1; c++) {
            const float4 a = ld_dep(reinterpret_cast<const float4 *>(src + (c - c0) * step));
            v.x += a.x; v.y += a.y; v.z += a.z; v.w += a.w;
        }
        const size_t at = (size_t)(n0 + t) * o.out_ld + o.out_row0 + row0;
        if constexpr (VEC) {
            if (row0 + 4 * lane < o.m)
                for (uint32_t b = 0; b < o.nout; b++) *reinterpret_cast<float4 *>(reinterpret_cast<OT *>(o.outs[b]) + at + 4 * lane) = v;
        } else {
            float e[4];  // rows lane, lane + 32, ..
#pragma unroll
            for (uint32_t j = 0; j < 4; j++) {
                const uint32_t from = 8 * j + lane / 4;
                const float x = __shfl_sync(0xffffffffu, v.x, from), y = __shfl_sync(0xffffffffu, v.y, from);
                const float z = __shfl_sync(0xffffffffu, v.z, from), w = __shfl_sync(0xffffffffu, v.w, from);
                e[j] = lane & 2 ? (lane & 1 ? w : z) : (lane & 1 ? y : x);
            }
            for (uint32_t b = 0; b < o.nout; b++) {
                OT *out = reinterpret_cast<OT *>(o.outs[b]) + at + lane;
#pragma unroll
                for (uint32_t j = 0; j < 4; j++)
                    if (row0 + lane + 32 * j < o.m) {
                        if constexpr (sizeof(OT) == 4) out[32 * j] = e[j];
                        else out[32 * j] = __float2bfloat16_rn(e[j]);
                    }
            }
        }
    }
}

template <int TY, int XDT, typename OT, int NACC>
static cudaError_t launch_n(const Args &a, const Outs &go, cudaStream_t s, int sms, int dev) {
    static bool attr_set[64] = {};  // the opt-in is per device
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (!attr_set[dev]) {
        cudaError_t e = cudaFuncSetAttribute(gemm_tc_kernel<TY, XDT, OT, NACC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Rings<TY, NACC>::smem);
        if (e != cudaSuccess) return e;
        attr_set[dev] = true;
    }
    const uint32_t groups = (a.n + NACC * kBN - 1) / (NACC * kBN), items = ((a.m + kBM - 1) / kBM) * groups;
    const uint32_t grid = a.waves ? (uint32_t)sms : a.dealt ? a.dealers : items < (uint32_t)sms ? items : (uint32_t)sms;
    alignas(64) CUtensorMap xmap;
    memset(&xmap, 0, sizeof(xmap));
    if constexpr (XDT != DT_F32) {
        cudaError_t me = encode_x_map(&xmap, a.x, a.k, a.n, kBN);
        if (me != cudaSuccess) return me;
    }
    return launch_pdl(gemm_tc_kernel<TY, XDT, OT, NACC>, grid, kThreads, Rings<TY, NACC>::smem, s, 1, xmap, a, go);
}

template <int TY, int XDT, typename OT>
static cudaError_t launch(const Args &a, const Outs &go, cudaStream_t s, int sms, int dev) {
    return launch_n<TY, XDT, OT, XDT == DT_F32 ? 1 : 2>(a, go, s, sms, dev);
}

template <int TY, int XDT>
static cudaError_t launch_o(const Args &a, const Outs &go, int odt, cudaStream_t s, int sms, int dev) {
    if (odt == DT_F32 && go.epoch) return launch<TY, XDT, GatherF32>(a, go, s, sms, dev);
    if (odt == DT_F32) return launch<TY, XDT, float>(a, go, s, sms, dev);
    if (odt == DT_BF16) return launch<TY, XDT, __nv_bfloat16>(a, go, s, sms, dev);
    return cudaErrorInvalidValue;
}

template <int TY>
static cudaError_t launch_x(const Args &a, const Outs &go, int xdt, int odt, cudaStream_t s, int sms, int dev) {
    switch (xdt) {
    case DT_F16: return launch_o<TY, DT_F16>(a, go, odt, s, sms, dev);
    case DT_BF16: return launch_o<TY, DT_BF16>(a, go, odt, s, sms, dev);
    case DT_F32: return launch_o<TY, DT_F32>(a, go, odt, s, sms, dev);
    default: return cudaErrorInvalidValue;
    }
}

// `tok`, `steps`: tokens of an item and what its k is dealt by
static cudaError_t launch_reduce(const float *part, const Args &a, const Outs &go, uint32_t tok, uint32_t steps, int odt, cudaStream_t s) {
    const uint32_t groups = (a.n + tok - 1) / tok, items = (a.m + kBM - 1) / kBM * groups;
    ReduceOut ro = {go.nout, a.m, a.n, go.out_ld, go.out_row0, a.dealt, items, steps, a.dealers, a.nt, groups, tok, {}, go.epoch, go.epoch_inc};
    bool vec = ((a.m | go.out_ld | go.out_row0) & 3) == 0;
    for (uint32_t o = 0; o < go.nout; o++) {
        ro.outs[o] = go.outs[o];
        vec = vec && (uintptr_t)go.outs[o] % 16 == 0;
    }
    const unsigned blocks = a.dealt * ((a.nt + kReduceTok - 1) / kReduceTok);
    if (odt == DT_BF16) return launch_pdl(reduce_kernel<__nv_bfloat16, false>, blocks, 256, kReduceSmem, s, 1, part, ro);
    if (vec) return launch_pdl(reduce_kernel<float, true>, blocks, 256, kReduceSmem, s, 1, part, ro);
    return launch_pdl(reduce_kernel<float, false>, blocks, 256, kReduceSmem, s, 1, part, ro);
}

}  // namespace tc

// fp32 activations -> bf16, once for all slabs, so that they come by TMA like the others.
__global__ void __launch_bounds__(256) to_bf16_kernel(const float4 *x, uint4 *__restrict__ y, size_t n8) {
    pdl_launch_dependents();
    pdl_wait();
    const float4 *in = dep_ptr(x);
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n8; i += (size_t)gridDim.x * blockDim.x) {
        const float4 a = ld_dep(in + 2 * i), b = ld_dep(in + 2 * i + 1);
        y[i] = make_uint4(tc::pack16<false>(a.x, a.y), tc::pack16<false>(a.z, a.w), tc::pack16<false>(b.x, b.y), tc::pack16<false>(b.z, b.w));
    }
}
cudaError_t launch_to_bf16(const void *x, void *y, size_t count, int sms, cudaStream_t s) {
    const size_t blocks = (count / 8 + 255) / 256, most = (size_t)sms * 8;
    return launch_pdl(to_bf16_kernel, (unsigned)(blocks < most ? blocks : most), 256, 0, s, 1, (const float4 *)x, (uint4 *)y, count / 8);
}

bool gemm_tc_supported(int ty, uint32_t k, uint32_t m, const void *w, const void *x, int xdt, uint32_t n) {
    if (!has_fast_kernels(ty)) return false;
    if (k % 64 || m == 0 || n == 0) return false;
    if ((uintptr_t)x % 16 || (k * (xdt == DT_F32 ? 4 : 2)) % 16) return false;
    if (ty == T_Q4_K && (uintptr_t)w % 16) return false;
    return true;
}

cudaError_t launch_gemm_tc(const GemmPlan &plan, int ty, const uint8_t *w, uint32_t k, uint32_t m, const void *x, int xdt,
                           uint32_t n, void *out, int odt, int *status, float *partial, cudaStream_t s, int sms, int dev,
                           uint64_t *launches, const GemvGatherPlan *gather) {
    tc::Args a = {};
    a.w = w; a.x = x; a.out = out; a.status = status; a.k = k; a.m = m; a.n = n;
    tc::Outs go = {};
    if (gather) {
        // row shards: the epilogue (or the reduction) stores into every rank's whole output
        go.nout = gather->nranks;
        go.out_ld = gather->seg[0].m_total;
        go.out_row0 = gather->seg[0].row_first;
        for (uint32_t r = 0; r < gather->nranks; r++) go.outs[r] = gather->seg[0].out[r];
        go.epoch = gather->epoch;
        go.epoch_inc = gather->nranks;
    } else {
        go.nout = 1; go.out_ld = m; go.out_row0 = 0; go.outs[0] = out;
    }
    a.waves = plan.waves; a.dealt = plan.dealt; a.dealers = plan.dealers; a.nt = plan.nt;
    a.partial = partial;
    *launches += plan.dealt ? 2 : 1;
    a.row_bytes = (k / block_elems(ty)) * block_bytes(ty);
    cudaError_t e = cudaErrorInvalidValue;
    if (plan.tok) {
        GemmTs g = {ty, xdt, odt, sms, w, x, out, status, partial, k, m, n, a.row_bytes, plan.tok, a.waves, a.dealt, a.dealers, a.nt, plan.cluster, plan.chains,
                    gather ? go.nout : 0u, go.out_ld, go.out_row0, {}, go.epoch, go.epoch_inc};
        for (uint32_t r = 0; r < go.nout; r++) g.outs[r] = go.outs[r];
        e = launch_gemm_ts(g, s, dev);
    } else {
        switch (ty) {
        case T_Q4_K: e = tc::launch_x<T_Q4_K>(a, go, xdt, odt, s, sms, dev); break;
        case T_Q8_0: e = tc::launch_x<T_Q8_0>(a, go, xdt, odt, s, sms, dev); break;
        case T_Q4_0: e = tc::launch_x<T_Q4_0>(a, go, xdt, odt, s, sms, dev); break;
        case T_Q6_K: e = tc::launch_x<T_Q6_K>(a, go, xdt, odt, s, sms, dev); break;
        case T_Q5_K: e = tc::launch_x<T_Q5_K>(a, go, xdt, odt, s, sms, dev); break;
        case T_IQ4_NL: e = tc::launch_x<T_IQ4_NL>(a, go, xdt, odt, s, sms, dev); break;
        case T_Q2_0: e = tc::launch_x<T_Q2_0>(a, go, xdt, odt, s, sms, dev); break;
        case T_IQ2_XXS: e = tc::launch_x<T_IQ2_XXS>(a, go, xdt, odt, s, sms, dev); break;
        }
    }
    if (e != cudaSuccess || !a.dealt) return e;
    return tc::launch_reduce(partial, a, go, plan.tok ? plan.tok : plan.nacc * tc::kBN, plan.tok ? (k + 255) / 256 : k / tc::kBK, odt, s);
}

}  // namespace okf

// ---- matmul without any allocation ----------------------------------------------------
// okf_gemm_noalloc serves callers that must not allocate device memory while they
// run: code inside a CUDA-graph capture or a real-time decode loop, a process that
// shares the GPU under a fixed memory budget, a plugin host that forbids cudaMalloc
// after start-up.  A matmul with dealt items normally takes its buffer of partial tiles from
// the context, which grows it with cudaMalloc on demand; here the buffer is a
// fixed array that is part of the loaded library image instead.
namespace okf {
constexpr size_t kStaticScratchFloats = (size_t)4 << 20;  // 16 MiB on every GPU that loads the library
static __device__ __align__(256) float g_static_scratch[kStaticScratchFloats];
// In host code the name above is only a stand-in for the symbol; the device address has
// to be asked for, once per device, with that device current.  The cache is not
// synchronised: two threads that meet here for the first time both look the address
// up and both store the same value.
static float *g_static_scratch_addr[64] = {};
}  // namespace okf

extern "C" int okf_gemm_noalloc(okf_ctx *ctx, int type, const okf_weights *w, uint64_t woff, uint32_t k, uint32_t m,
                                const void *x, int xdt, uint32_t n, void *out, int odt, okf_stream stream) {
    using namespace okf;
    int rc = check_gemm_args(ctx, type, w, woff, k, m, x, xdt, n, out, odt);
    if (rc) return rc;
    const uint8_t *wp = w->dptr + woff;
    if (!gemm_tc_supported(type, k, m, wp, x, xdt, n)) return OKF_E_ALIGN;
    if (k / tc::kBK < 2) return OKF_E_SHAPE;
    if (2 * (size_t)n * m > kStaticScratchFloats) return OKF_E_LIMIT;  // N * M above 2 Mi outputs
    if (fault_fires(ctx)) return OKF_E_INJECTED;
    DeviceGuard g(ctx->device);
    if (!g.ok) return cuda_fail(ctx, cudaErrorInvalidDevice);
    if (ctx->device < 0 || ctx->device >= 64) return OKF_E_ARG;
    if (!g_static_scratch_addr[ctx->device]) {
        // first call on this device: resolve the array's device address
        float *ptr = nullptr;
        cudaError_t e = cudaGetSymbolAddress((void **)&ptr, g_static_scratch);
        if (e != cudaSuccess) return cuda_fail(ctx, e);
        g_static_scratch_addr[ctx->device] = ptr;
    }
    // every slot the reduction reads is written by the main kernel first, so nothing in the
    // array has to be cleared between calls
    const GemmPlan plan = gemm_tc_plan(type, k, m, n, xdt, ctx->sms, kStaticScratchFloats,
                                       ctx->flags & OKF_FLAG_DEAL_ITEMS ? nullptr : gemm_ts_clusters(ctx->device));
    cudaError_t e = launch_gemm_tc(plan, type, wp, k, m, x, xdt, n, out, odt, ctx->dev_status, g_static_scratch_addr[ctx->device],
                                   (cudaStream_t)stream, ctx->sms, ctx->device, &ctx->launches, nullptr);
    if (e != cudaSuccess) return cuda_fail(ctx, e);
    return OKF_OK;
}
