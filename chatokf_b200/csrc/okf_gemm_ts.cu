// Prefill matmul whose weight operand goes through tensor memory: out[n][m] = sum_k X[n][k] W[m][k] for N >= 9
// tokens of 16-bit activations, up to 256 tokens at a time.
//
// With few tokens to a weight the time goes into unpacking.  In okf_gemm_tc.cu every k-block of 128 rows x 64 k
// passes through the L1 / shared-memory pipe three times: 16-byte loads of sixteen rows a warp apart (a look-up a
// row each), the unpacked 16 KB into shared memory, and out of it again by the tensor core; 0.42 us per k-block whatever the
// tokens.  Here
//   - blocks come as stored (128 rows x 256 k, a "unit") into a ring in shared memory by 2-D TMA, rows an odd number of
//     16 bytes apart so that a warp reads 32 rows without conflicts;
//   - sixteen warps unpack: thread = row, warp = 32 rows (the quarter of tensor memory it may touch) x two of a
//     unit's four k-blocks; two sets of eight warps take the units in turn;
//   - 64 weights leave as 32 registers with one tcgen05.st, and tcgen05.mma takes its A operand from there:
//     tensor memory holds the accumulator(s) in columns 0 .. 255 and a unit of weights per set in 256 .. 511;
//   - activation tiles arrive by TMA, one warp issues the MMAs, a unit a turn, four run the epilogue, as in okf_gemm_tc.cu.
// 5120 -> 17408, 64 tokens, us, there and here: Q8_0 47.6 -> 26.1, Q4_0 37.9 -> 22.7, Q6_K 59.9 -> 29.4, Q4_K 37.6 -> 23.4,
// IQ2_XXS 38.1 -> 25.0, IQ4_NL 40.8 -> 27.6; Q5_K 2560 -> 9728, 77 tokens, 19.3 -> 14.8.  What bounds it: up to some 100 tokens instruction issue
// (about 260 instructions for a warp's 32 x 64 weights: widening, multiply-add, rounding; 58 % of the issue slots for Q4_K at 64 tokens, 68 % for
// IQ2_XXS); at 256 tokens nothing is full, the tensor pipe is busy 55 % of the time and a third of the slots are used.
// Where there are few items (a short prompt against few rows), clusters of 2 to 8 CTAs share one: each takes a run of its units, leaves its sums in
// shared memory where the rings were, and adds up every so many-th token out of the others' (share_out in okf_gemm_plan.h has what it
// gives: 1.1 to 2 times on the shapes that take it, against partial tiles through L2 and a second kernel).
// Tried on the way: rows copied by cp.async (two warps: 1900 cycles a unit for address arithmetic and issue, Q4_K 30.8 us against 25.9);
// a turn of the MMA warp per k-block (some 500 cycles each, 28.9); one k-block a turn for every unpacking warp (25.9
// against 23.0: waits and stores are paid per turn).
//
// Every wait is bounded (about a second); a wait that gives up records a code in the status word.
#include <cstring>
#include <mutex>

#include "okf_tc.cuh"
#include "okf_gemv_wide.cuh"
#include "okf_gemm_ts.h"
#include "okf_kernels.h"
#include "okf_ring.h"

namespace okf {
namespace tc {

constexpr uint32_t kTsUnpackWarps = 16, kTsSetWarps = 8;  // two sets, a unit each in turn
constexpr uint32_t kTsTmaWarp = 16, kTsMmaWarp = 17, kTsLoadWarp = 18;  // loaders: 18, 19; epilogue: 20 .. 23
constexpr uint32_t kTsThreads = 24 * 32;
constexpr uint32_t kTsACol = 256, kTsACols = 128;  // a unit of weights: four k-blocks of 32 columns
constexpr uint32_t kTsMaxW = 8, kTsMaxB = 12;
constexpr uint32_t kTsBarBytes = 512;
constexpr uint32_t kTsSmem = 225 * 1024;  // of 227
constexpr uint32_t kTsTabCopies = 32;     // IQ2_XXS: look-ups without bank conflicts, see Iq2Tab

// Geometry of a unit (256 k of a row) in the ring: rows an odd number of 16 bytes apart.  SK: what is copied starts at the
// 16- (TMA) or 8-byte boundary (cp.async) below the unit, which may lie on any 2-byte boundary.  Without SK every row starts on 16
// bytes, so a tensor map describes them.
template <int TY, bool SK> struct TsGeom {
    static constexpr uint32_t ub = Geom<TY>::bytes * (256 / Geom<TY>::per);
    static constexpr uint32_t cp = 8, need = (ub + 6 + cp - 1) / cp;  // cp.async: bytes of a piece, pieces of a row
    static constexpr uint32_t rs = ((ub + (SK ? 14 : 0) + 15) / 16 | 1) * 16;
    static constexpr uint32_t stage = kBM * rs;
};

struct TsArgs {
    const uint8_t *w;
    void *out;
    int *status;
    float *partial;
    uint32_t k, m, n, row_bytes;
    uint32_t tok, groups, items;         // tokens of an item (a multiple of 16), items per slab, all items
    uint32_t waves, dealt, dealers, nt;  // as in okf_gemm_tc.cu, but dealt by units
    uint32_t w_stages, b_stages, box, b_kb, b_off, w_off, tab_off;  // a stage of activations: box tokens x b_kb k-blocks of a unit
    uint32_t tma_log;  // weights by TMA, 2^tma_log rows to a row of the tensor map; kTsNoTma: by cp.async
    uint32_t odt;      // DT_F32, DT_BF16
    uint32_t cluster;  // CTAs that share an item along K (<= 1: none)
    uint32_t chains;   // shared items: accumulators that take k-blocks in turn (1, 2 or 4)
    uint32_t vec;      // shared items: rows of results start on 16 (bf16: 8) bytes
    uint32_t nout, out_ld, out_row0;  // row shards: fp32 into every rank's whole output (nout > 0)
    void *outs[8];
    uint32_t *epoch;
    uint32_t epoch_inc;
};

struct TsWork {
    uint32_t m0, n0, kb0, kb1;
    uint32_t slot;  // partial tile, or kTsWhole, or kTsShare
};
constexpr uint32_t kTsWhole = 0xFFFFFFFFu, kTsShare = 0xFFFFFFFEu, kTsNoTma = 0xFFFFFFFFu;

// The j-th piece of work of this CTA; false when there is none.  Whole items go round-robin over the CTAs, then every CTA
// takes its run of the dealt items' units laid end to end (the CTA that has a unit: dealt_to).
// CL: one item a cluster, this CTA's part of its K.
template <bool CL> __device__ __forceinline__ bool ts_work(const TsArgs &p, uint32_t j, TsWork &w) {
    const uint32_t kblocks = p.k / kBK, units = (kblocks + 3) / 4;
    uint32_t item;
    w.slot = kTsWhole;
    w.kb0 = 0;
    w.kb1 = kblocks;
    if constexpr (CL) {
        if (j) return false;
        item = blockIdx.x / p.cluster;
        const uint32_t rank = blockIdx.x - item * p.cluster;
        w.kb0 = units * rank / p.cluster * 4;
        w.kb1 = min(units * (rank + 1) / p.cluster * 4, kblocks);
        w.slot = kTsShare;
    } else if (!p.dealt || j < p.waves) {
        item = blockIdx.x + j * gridDim.x;
        if (item >= p.items) return false;
    } else {
        const uint32_t total = p.dealt * units;
        if (blockIdx.x >= p.dealers) return false;
        const uint32_t lo = total * blockIdx.x / p.dealers, hi = total * (blockIdx.x + 1) / p.dealers;
        const uint32_t i = lo / units + (j - p.waves), start = max(lo, i * units), end = min(hi, (i + 1) * units);
        if (start >= end) return false;
        w.kb0 = (start - i * units) * 4;
        w.kb1 = min((end - i * units) * 4, kblocks);
        if (end - start < units) w.slot = (blockIdx.x - dealt_to(i * units, total, p.dealers)) * p.dealt + i;
        item = p.items - p.dealt + i;
    }
    const uint32_t slab = item / p.groups;
    w.m0 = slab * kBM;
    w.n0 = (item - slab * p.groups) * p.tok;
    return true;
}

__device__ __forceinline__ void cp_async8(uint32_t dst, const uint8_t *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
// this thread's copies so far arrive on the barrier when they have landed (the barrier counts the threads)
__device__ __forceinline__ void cp_async_arrive(uint64_t *bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
          "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]),
          "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]),
          "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// A from tensor memory: lane = row, a column = two consecutive k
__device__ __forceinline__ void umma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// ---- an item that the CTAs of a cluster share ----------------------------------------
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// 16 bytes of CTA `rank`'s shared memory, at the place that `addr` is in this one's
__device__ __forceinline__ float4 lds_of(uint32_t addr, uint32_t rank) {
    float4 v;
    asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %4, %5;\n\tld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [a];\n\t}"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr), "r"(rank) : "memory");
    return v;
}
// Rows m0 + 4 lane .. + 3 of token `t`, into every output.  Where results do not start on 16 (8) bytes the neighbours of every thread are dealt out
// again, so that a warp stores 32 rows side by side.
__device__ __forceinline__ void store_rows(const TsArgs &p, float4 v, uint32_t m0, uint32_t t, uint32_t lane) {
    const size_t at = (size_t)t * (p.nout ? p.out_ld : p.m) + (p.nout ? p.out_row0 : 0u) + m0;
    float e[4];  // rows lane, lane + 32, ..
    if (!p.vec) {
#pragma unroll
        for (uint32_t j = 0; j < 4; j++) {
            const uint32_t from = 8 * j + lane / 4;
            const float x = __shfl_sync(0xffffffffu, v.x, from), y = __shfl_sync(0xffffffffu, v.y, from);
            const float z = __shfl_sync(0xffffffffu, v.z, from), w = __shfl_sync(0xffffffffu, v.w, from);
            e[j] = lane & 2 ? (lane & 1 ? w : z) : (lane & 1 ? y : x);
        }
    }
#pragma unroll 1
    for (uint32_t b = 0; b < (p.nout ? p.nout : 1u); b++) {
        void *out = p.nout ? p.outs[b] : p.out;
        if (p.vec) {
            if (m0 + 4 * lane >= p.m) break;
            if (p.odt == DT_F32) *reinterpret_cast<float4 *>(reinterpret_cast<float *>(out) + at + 4 * lane) = v;
            else *reinterpret_cast<uint2 *>(reinterpret_cast<__nv_bfloat16 *>(out) + at + 4 * lane) = make_uint2(pack16<false>(v.x, v.y), pack16<false>(v.z, v.w));
        } else {
#pragma unroll
            for (uint32_t j = 0; j < 4; j++) {
                if (m0 + lane + 32 * j >= p.m) continue;
                if (p.odt == DT_F32) reinterpret_cast<float *>(out)[at + lane + 32 * j] = e[j];
                else reinterpret_cast<__nv_bfloat16 *>(out)[at + lane + 32 * j] = __float2bfloat16_rn(e[j]);
            }
        }
    }
}

// ---- unpacking 64 weights of a row ------------------------------------------------
// A code becomes a float without the integer pipe's byte permutes and conversions: the code bytes of a word, two to a
// register and 16 bits apart, are fp16 subnormals (code x 2^-24) as they stand, and widening them is an instruction of the
// floating-point pipe.  The 2^24 goes into the scale, which stays exact; so weights are decoded in fp32, mul * code + add, as
// the reference decodes them, and rounded once.
struct Affine {  // mul * 2^24 and add, twice each: fma.rn.f32x2 takes two weights at a time
    uint64_t mul, add;
    __device__ __forceinline__ Affine(float m, float a) {
        m *= 16777216.f;
        asm("mov.b64 %0, {%1, %1};" : "=l"(mul) : "f"(m));
        asm("mov.b64 %0, {%1, %1};" : "=l"(add) : "f"(a));
    }
};
template <bool F16>
__device__ __forceinline__ uint32_t scale2(float a, float b, const Affine &t) {
    float x, y;
    asm("{\n\t.reg .b64 v;\n\tmov.b64 v, {%2, %3};\n\tfma.rn.f32x2 v, v, %4, %5;\n\tmov.b64 {%0, %1}, v;\n\t}"
        : "=f"(x), "=f"(y) : "f"(a), "f"(b), "l"(t.mul), "l"(t.add));
    return pack16<F16>(x, y);
}
// weights k .. k + 3 out of codes (k, k + 2) and (k + 1, k + 3), sixteen bits each
template <bool F16>
__device__ __forceinline__ void halves4(uint32_t even, uint32_t odd, const Affine &t, uint32_t *o) {
    const float2 e = __half22float2(*reinterpret_cast<const __half2 *>(&even)), f = __half22float2(*reinterpret_cast<const __half2 *>(&odd));
    o[0] = scale2<F16>(e.x, f.x, t);
    o[1] = scale2<F16>(e.y, f.y, t);
}
// two neighbours
template <bool F16>
__device__ __forceinline__ uint32_t pair(uint32_t w, const Affine &t) {
    const float2 e = __half22float2(*reinterpret_cast<const __half2 *>(&w));
    return scale2<F16>(e.x, e.y, t);
}
// the four bytes of a word
template <bool F16>
__device__ __forceinline__ void codes4(uint32_t w, const Affine &t, uint32_t *o) {
    halves4<F16>(w & 0x00FF00FFu, prmt(w, 0u, 0x4341u), t, o);
}

// 4 * NW bytes of a row in shared memory; SK: at a 2-byte boundary, else a 4-byte one (16 bytes at a time where
// NW is a multiple of four: such pieces start on 16-byte boundaries)
template <int NW, bool SK>
__device__ __forceinline__ void row_words(uint32_t a, uint32_t (&v)[NW]) {
    if constexpr (SK) {
        lds_a2<NW>(a, v);
    } else if constexpr (NW % 4 == 0) {
#pragma unroll
        for (int i = 0; i < NW / 4; i++) {
            const uint4 q = lds128(a + 16 * i);
            v[4 * i] = q.x; v[4 * i + 1] = q.y; v[4 * i + 2] = q.z; v[4 * i + 3] = q.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < NW; i++) v[i] = lds32(a + 4 * i);
    }
}
// At a 2-byte boundary in 8-byte words, for types that need many: a warp's 4-byte words of one column of rows 16 bytes
// (times an odd number) apart meet four to a bank.
template <int NW>
__device__ __forceinline__ void words8(uint32_t a, uint32_t (&v)[NW]) {
    const uint32_t base = a & ~7u, sh = (a & 2u) * 8u;
    uint32_t w[NW + 4];
#pragma unroll
    for (int i = 0; i < NW / 2 + 1; i++) {
        const uint2 q = lds64(base + 8 * i);
        w[2 * i] = q.x;
        w[2 * i + 1] = q.y;
    }
    w[NW + 2] = w[NW + 1];
    const bool odd = a & 4u;
#pragma unroll
    for (int i = 0; i <= NW; i++) w[i] = odd ? w[i + 1] : w[i];
#pragma unroll
    for (int i = 0; i < NW; i++) v[i] = __funnelshift_r(w[i], w[i + 1], sh);
}

// What one thread takes out of the ring for k-block `p` of the unit at `a`; unpack() writes its 64 weights as
// pairs in order of k.
template <int TY, bool SK> struct TsRaw;
// Q4_K, Q5_K: 32 bytes of qs; low nibbles are sub-block 2p, high ones 2p + 1 (LLM/Quantize/KQuants.swift:104-158)
template <int TY, bool SK> struct TsRawK45 {
    uint32_t h[4], q[8], f[TY == T_Q5_K ? 8 : 1];
    __device__ __forceinline__ void load(uint32_t a, uint32_t p) {
        row_words<4, SK>(a, h);
        if constexpr (TY == T_Q5_K) row_words<8, SK>(a + 16, f);
        row_words<8, SK>(a + (TY == T_Q4_K ? 16 : 48) + 32 * p, q);
    }
    template <bool F16> __device__ __forceinline__ void unpack(uint32_t p, const Iq2Tab &, uint32_t (&o)[32]) const {
        // 6-bit scales and mins of sub-blocks 2p and 2p + 1 (get_scale_min_k4): bytes 2p, 2p + 1 of the
        // scale field for p < 2, split fields above
        const uint32_t sh = (p & 1) * 16, a = h[1] >> sh, b = h[2] >> sh, e = h[3] >> sh;
        const uint32_t sc = p < 2 ? a & 0x3F3Fu : (e & 0x0F0Fu) | ((a >> 2) & 0x3030u);
        const uint32_t mn = p < 2 ? b & 0x3F3Fu : ((e >> 4) & 0x0F0Fu) | ((b >> 2) & 0x3030u);
        const float d = f16bits(h[0] & 0xFFFF), dm = f16bits(h[0] >> 16);
        const float d0 = d * byte_to_f32(sc, 0), d1 = d * byte_to_f32(sc, 1);
        // Q4_K's high nibbles stay where they are, 16 x the code
        const Affine t0(d0, -dm * byte_to_f32(mn, 0)), t1(TY == T_Q4_K ? d1 * 0.0625f : d1, -dm * byte_to_f32(mn, 1));
#pragma unroll
        for (int i = 0; i < 8; i++) {
            if constexpr (TY == T_Q4_K) {
                const uint32_t w = q[i], v = w >> 8;
                halves4<F16>(w & 0x000F000Fu, v & 0x000F000Fu, t0, o + 2 * i);
                halves4<F16>(w & 0x00F000F0u, v & 0x00F000F0u, t1, o + 16 + 2 * i);
            } else {
                const uint32_t t = f[i] >> (2 * p);
                codes4<F16>((q[i] & 0x0F0F0F0Fu) | ((t << 4) & 0x10101010u), t0, o + 2 * i);
                codes4<F16>(((q[i] >> 4) & 0x0F0F0F0Fu) | ((t << 3) & 0x10101010u), t1, o + 16 + 2 * i);
            }
        }
    }
};
template <bool SK> struct TsRaw<T_Q4_K, SK> : TsRawK45<T_Q4_K, SK> {};
template <bool SK> struct TsRaw<T_Q5_K, SK> : TsRawK45<T_Q5_K, SK> {};
// Q6_K: granules 2 (p & 1) and the next of half p / 2: 64 bytes of ql (low nibbles for even p), two bits each of 32
// bytes of qh, four scales (LLM/Quantize/KQuants.swift:160-177)
template <> struct TsRaw<T_Q6_K, true> {
    uint32_t l[16], g[8], sc, d;
    __device__ __forceinline__ void load(uint32_t a, uint32_t p) {
        words8<16>(a + 64 * (p >> 1), l);
        words8<8>(a + 128 + 32 * (p >> 1), g);
        uint32_t s[1];
        lds_a2<1>(a + 192 + 4 * p, s);
        sc = s[0];
        d = lds16(a + 208);
    }
    template <bool F16> __device__ __forceinline__ void unpack(uint32_t p, const Iq2Tab &, uint32_t (&o)[32]) const {
        const float df = f16bits(d);
        const uint32_t sh = 4 * (p & 1);
#pragma unroll
        for (int i = 0; i < 4; i++) {  // sixteen weights, one scale
            const float m = df * (float)(int)(int8_t)(sc >> (8 * i) & 0xFF);
            const Affine t(m, -32.f * m);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const uint32_t b = g[4 * (i & 1) + j] >> sh;
                codes4<F16>(((l[4 * i + j] >> sh) & 0x0F0F0F0Fu) | ((i < 2 ? b << 4 : b << 2) & 0x30303030u), t, o + 8 * i + 2 * j);
            }
        }
    }
};
// Q8_0: two blocks {f16 d; i8 q[32]} (LLM/Gemma/Gemma4Quant.swift:51-69)
template <bool SK> struct TsRaw<T_Q8_0, SK> {
    uint32_t w[17];
    __device__ __forceinline__ void load(uint32_t a, uint32_t p) { row_words<17, SK>(a + 68 * p, w); }
    template <bool F16> __device__ __forceinline__ void unpack(uint32_t, const Iq2Tab &, uint32_t (&o)[32]) const {
        const float d0 = f16bits(w[0] & 0xFFFF), d1 = f16bits(w[8] >> 16);
#pragma unroll
        for (int b = 0; b < 2; b++) {
            const Affine t(b ? d1 : d0, -128.f * (b ? d1 : d0));
#pragma unroll
            for (int j = 0; j < 8; j++)  // the first block's quants start two bytes into word 0, the second's on word 9
                codes4<F16>((b ? w[9 + j] : __funnelshift_r(w[j], w[j + 1], 16)) ^ 0x80808080u, t, o + 16 * b + 2 * j);  // q + 128
        }
    }
};
// Q4_0, IQ4_NL: two blocks {f16 d; u8 qs[16]}, byte j = weights j (low nibble) and j + 16 (LLM/Gemma/Gemma4Quant.swift:5-49)
template <int TY, bool SK> struct TsRaw40 {
    uint32_t w[9];
    __device__ __forceinline__ void load(uint32_t a, uint32_t p) { row_words<9, SK>(a + 36 * p, w); }
    template <bool F16> __device__ __forceinline__ void unpack(uint32_t, const Iq2Tab &, uint32_t (&o)[32]) const {
#pragma unroll
        for (int b = 0; b < 2; b++) {
            const float d = f16bits(b ? w[4] >> 16 : w[0] & 0xFFFF);
            const Affine t(d, (TY == T_Q4_0 ? -8.f : -128.f) * d), th(0.0625f * d, -8.f * d);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t q = b ? w[5 + i] : __funnelshift_r(w[i], w[i + 1], 16);
                if constexpr (TY == T_Q4_0) {
                    const uint32_t v = q >> 8;
                    halves4<F16>(q & 0x000F000Fu, v & 0x000F000Fu, t, o + 16 * b + 2 * i);
                    halves4<F16>(q & 0x00F000F0u, v & 0x00F000F0u, th, o + 16 * b + 8 + 2 * i);
                } else {
                    // the codebook's values + 128, looked up eight nibbles a word (see iq4nl_word): t0 holds those of
                    // bytes 0 and 1 (low, high, low, high), t1 those of bytes 2 and 3
                    constexpr uint32_t T0 = 0x3F2D1801u, T1 = 0x766A5D4Fu, T2 = 0xA6998D81u, T3 = 0xF1D9C5B5u;
                    const uint32_t sel = q & 0x77777777u, pick = (q >> 1 & 0x44444444u) | 0x32103210u;
                    const uint32_t t0 = prmt(prmt(T0, T1, sel), prmt(T2, T3, sel), pick);
                    const uint32_t t1 = prmt(prmt(T0, T1, sel >> 16), prmt(T2, T3, sel >> 16), pick >> 16);
                    o[16 * b + 2 * i] = pair<F16>(t0 & 0x00FF00FFu, t);
                    o[16 * b + 2 * i + 1] = pair<F16>(t1 & 0x00FF00FFu, t);
                    o[16 * b + 8 + 2 * i] = pair<F16>(prmt(t0, 0u, 0x4341u), t);
                    o[16 * b + 8 + 2 * i + 1] = pair<F16>(prmt(t1, 0u, 0x4341u), t);
                }
            }
        }
    }
};
template <bool SK> struct TsRaw<T_Q4_0, SK> : TsRaw40<T_Q4_0, SK> {};
template <bool SK> struct TsRaw<T_IQ4_NL, SK> : TsRaw40<T_IQ4_NL, SK> {};
// Q2_0: half p & 1 of block p / 2, {f16 d; u8 qs[32]} of 128 codes, weight = (code - 1) * d (LLM/Base/Quant.swift:2-25)
template <> struct TsRaw<T_Q2_0, true> {
    uint32_t w[4], d;
    __device__ __forceinline__ void load(uint32_t a, uint32_t p) {
        d = lds16(a + 34 * (p >> 1));
        lds_a2<4>(a + 34 * (p >> 1) + 2 + 16 * (p & 1), w);
    }
    template <bool F16> __device__ __forceinline__ void unpack(uint32_t, const Iq2Tab &, uint32_t (&o)[32]) const {
        const Affine t(f16bits(d), -f16bits(d));
#pragma unroll
        for (int i = 0; i < 4; i++) {
            // code e of every byte, then side by side: byte b of the word holds weights 4b .. 4b + 3
            uint32_t c[4];
#pragma unroll
            for (int e = 0; e < 4; e++) c[e] = w[i] >> (2 * e) & 0x03030303u;
            const uint32_t even01 = prmt(c[0], c[2], 0x5140u), odd01 = prmt(c[1], c[3], 0x5140u);
            const uint32_t even23 = prmt(c[0], c[2], 0x7362u), odd23 = prmt(c[1], c[3], 0x7362u);
            halves4<F16>(prmt(even01, 0u, 0x4140u), prmt(odd01, 0u, 0x4140u), t, o + 8 * i);
            halves4<F16>(prmt(even01, 0u, 0x4342u), prmt(odd01, 0u, 0x4342u), t, o + 8 * i + 2);
            halves4<F16>(prmt(even23, 0u, 0x4140u), prmt(odd23, 0u, 0x4140u), t, o + 8 * i + 4);
            halves4<F16>(prmt(even23, 0u, 0x4342u), prmt(odd23, 0u, 0x4342u), t, o + 8 * i + 6);
        }
    }
};
// IQ2_XXS: sub-blocks 2p and 2p + 1, {u32: four codebook indices, u32: four 7-bit sign indices + 4-bit scale}
// (LLM/Quantize/IQ2XXS.swift:34-53)
template <> struct TsRaw<T_IQ2_XXS, true> {
    uint32_t w[4], d;
    __device__ __forceinline__ void load(uint32_t a, uint32_t p) {
        d = lds16(a);
        lds_a2<4>(a + 2 + 16 * p, w);
    }
    template <bool F16> __device__ __forceinline__ void unpack(uint32_t, const Iq2Tab &tab, uint32_t (&o)[32]) const {
        constexpr uint32_t P = 0x406B5948u, N = 0x40152738u;  // 64 + {8, 25, 43, 0}, 64 - {8, 25, 43, 0}
        const float df = f16bits(d);
#pragma unroll
        for (int b = 0; b < 2; b++) {
            const uint32_t a0 = w[2 * b], a1 = w[2 * b + 1];
            const float db = df * (0.5f + (float)(a1 >> 28)) * 0.25f;
            const Affine t(db, -64.f * db);
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const uint32_t s = lds32(tab.code + prmt(a0, 0u, 0x4440 + c) * (kTsTabCopies * 4)) |
                                   lds32(tab.sign + (a1 >> (7 * c) & 127u) * (kTsTabCopies * 4));
                codes4<F16>(prmt(P, N, s), t, o + 16 * b + 4 * c);
                codes4<F16>(prmt(P, N, s >> 16), t, o + 16 * b + 4 * c + 2);
            }
        }
    }
};

// CL: launched in clusters that share an item along K.  (As a run-time flag it costs all other launches 0.3 us.)
template <int TY, bool SK, bool F16, bool CL>
__global__ void __launch_bounds__(kTsThreads, 1) gemm_ts_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap,
                                                               const __grid_constant__ TsArgs p) {
    using Ge = TsGeom<TY, SK>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t *full_w = reinterpret_cast<uint64_t *>(smem), *empty_w = full_w + 2 * kTsMaxW;  // loader <-> unpacking warps, see RingPlace
    uint64_t *full_a = empty_w + kTsMaxW, *empty_a = full_a + 2;                         // unpacking warps <-> MMA, one pair per set
    uint64_t *full_b = empty_a + 2, *empty_b = full_b + kTsMaxB;                         // TMA <-> MMA
    uint64_t *acc_full = empty_b + kTsMaxB, *acc_empty = acc_full + 2;                   // MMA <-> epilogue
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_empty + 2);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    static_assert((3 * kTsMaxW + 4 + 2 * kTsMaxB + 4) * 8 + 8 <= kTsBarBytes, "room for the barriers");

    const uint32_t warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;  // (uniform, and known to be)
    pdl_launch_dependents();
    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < p.w_stages; s++) {
            mbar_init(&full_w[s], p.tma_log == kTsNoTma ? 64 : 1);
            mbar_init(&full_w[p.w_stages + s], p.tma_log == kTsNoTma ? 64 : 1);
            mbar_init(&empty_w[s], kTsSetWarps);
        }
        for (uint32_t s = 0; s < 2; s++) {
            mbar_init(&full_a[s], kTsSetWarps);
            mbar_init(&empty_a[s], 1);
            mbar_init(&acc_full[s], 1);
            mbar_init(&acc_empty[s], 4);
        }
        for (uint32_t s = 0; s < p.b_stages; s++) {
            mbar_init(&full_b[s], 1);
            mbar_init(&empty_b[s], 1);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if constexpr (TY == T_IQ2_XXS) {
        uint32_t *tab = reinterpret_cast<uint32_t *>(smem + p.tab_off);
        // Sixteen entries a warp, worked out once and stored by all lanes side by side.  (Worked out anew for every copy, a
        // launch started 3 us later: 6144 -> 1500, 40 tokens, 17.4 us, so 13.6.)
        static_assert(kTsThreads / 32 * 16 == 384 && kTsTabCopies == 32, "entries to warps, copies to lanes");
        const uint32_t e = warp * 16 + (lane & 15), v = e < 256 ? iq2_code_selectors(g_iq2xxs_grid[e]) : iq2_sign_selectors(e - 256);
#pragma unroll
        for (uint32_t i = 0; i < 16; i++) tab[(warp * 16 + i) * kTsTabCopies + lane] = __shfl_sync(0xffffffffu, v, i);
    }
    if (warp == kTsMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    const uint32_t two_acc = p.tok <= 128 ? 1u : 0u;  // room for two accumulators
    // (a CTA of a cluster has five k-blocks at least, two units but for the last one's end: every accumulator gets one)
    const uint32_t chains = CL ? p.chains : 1, chain_cols = 256 / chains;

    TsWork wk;
    if (warp < kTsUnpackWarps) {
        // ---------------- unpack: row = 32 (warp % 4) + lane; two sets of eight warps take the units in turn, each with a stage
        // of tensor memory of its own; a warp has the k-blocks 2 kp and 2 kp + 1 of its unit
        const uint32_t row = (warp & 3) * 32 + lane, kp = warp >> 2 & 1, set = warp / kTsSetWarps;
        const uint32_t tl = p.tma_log == kTsNoTma ? 0 : p.tma_log, skew_mask = p.tma_log == kTsNoTma ? Ge::cp - 1 : 15u;
        const uint32_t slot = ((row & ((1u << tl) - 1)) << (7 - tl)) + (row >> tl);  // rows of one copy lie together
        const uint32_t ring = smem_u32(smem + p.w_off) + slot * Ge::rs;
        const uint32_t a_tmem = tmem_base + ((warp & 3) * 32 << 16) + kTsACol + set * kTsACols + kp * 64;
        Iq2Tab tab = {0, 0, 0};
        if constexpr (TY == T_IQ2_XXS) {
            tab.code = smem_u32(smem + p.tab_off) + lane * 4;
            tab.sign = tab.code + 256 * kTsTabCopies * 4;
        }
        RingPlace ring_at(set);
        uint32_t it = 0, turn = 0;  // units so far, of both sets and of this one
        for (uint32_t j = 0; ts_work<CL>(p, j, wk); j++) {
            const uint32_t src = (uint32_t)reinterpret_cast<uintptr_t>(p.w) + (wk.m0 + row) * p.row_bytes;  // its low bits
            for (uint32_t u = wk.kb0 >> 2; u < (wk.kb1 + 3) >> 2; u++, it++) {
                if ((it & 1) != set) continue;
                const uint32_t sw = ring_at.stage(p.w_stages);
                if (!warp_wait(&full_w[ring_at.full()], ring_at.full_parity(), lane, abort_flag, p.status)) goto done;
                const uint32_t at = ring + sw * Ge::stage + (SK ? (src + u * Ge::ub) & skew_mask : 0u);
                // does the tensor core still read this set's stage?  (the answer is there when the first weights are)
                const bool free_a = turn == 0 || mbar_test_wait(&empty_a[set], (turn - 1) & 1);
#pragma unroll
                for (uint32_t i = 0; i < 2; i++) {
                    const uint32_t q = 2 * kp + i;
                    const bool mine = 4 * u + q >= wk.kb0 && 4 * u + q < wk.kb1;
                    uint32_t v[32];
                    TsRaw<TY, SK> raw;
                    if (mine) raw.load(at, q);
                    if (mine) raw.template unpack<F16>(q, tab, v);
                    if (i == 0 && !__all_sync(0xffffffffu, free_a) &&
                        !warp_wait(&empty_a[set], (turn - 1) & 1, lane, abort_flag, p.status))
                        goto done;
                    if (mine) {
                        tc_fence_after();
                        tmem_st32(a_tmem + i * 32, v);
                    }
                }
                // The stage goes back only here, when every word loaded from it has been used: the copy that refills it waits
                // for this arrival and for nothing else.  (Handed back behind the second k-block's loads, with their words still
                // on the way, a row of Q8_0 2048 -> 5000, 700 tokens, once came out with one word of the next unit in it.)
                __syncwarp();
                if (lane == 0) mbar_arrive(&empty_w[sw]);
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&full_a[set]);
                turn++;
                ring_at.advance(2, p.w_stages);
            }
        }
    } else if (warp == kTsLoadWarp && p.tma_log != kTsNoTma) {
        // ---------------- blocks as stored -> ring; weights do not depend on the kernel before
        RingPlace ring_at(0);
        for (uint32_t j = 0; ts_work<CL>(p, j, wk); j++) {
            for (uint32_t u = wk.kb0 >> 2; u < (wk.kb1 + 3) >> 2; u++, ring_at.advance(1, p.w_stages)) {
                const uint32_t s = ring_at.stage(p.w_stages);
                uint64_t *full = &full_w[ring_at.full()];
                if (!ring_at.first_use(p.w_stages) && !warp_poll(&empty_w[s], ring_at.empty_parity(p.w_stages), abort_flag, p.status)) {
                    // giving up: the copies already handed over land within microseconds; stay for a
                    // while so that they do not write into a CTA that has gone
                    const long long t0 = clock64();
                    while (clock64() - t0 < 100000) {}
                    goto done;
                }
                if (elect_one()) {
                    mbar_expect_tx(full, Ge::stage);
                    for (uint32_t i = 0; i < 1u << p.tma_log; i++)
                        tma_load_tile(smem + p.w_off + s * Ge::stage + i * (Ge::stage >> p.tma_log), &wmap, ((i * p.row_bytes + u * Ge::ub) & ~15u) >> 2,
                                      wk.m0 >> p.tma_log, full);
                }
                __syncwarp();
            }
        }
    } else if (warp == kTsLoadWarp || warp == kTsLoadWarp + 1) {
        // ---------------- the same by cp.async, where rows are laid out so that a tensor map cannot describe them.
        // Eight lanes to a row, eight rows to a step of the two warps.  Every row of a unit copies the same number of pieces: what
        // that is too much lies inside the row's neighbour or the padding behind the last row.
        if constexpr (SK) if (p.tma_log == kTsNoTma) {
            const uint32_t first = (warp - kTsLoadWarp) * 4 + (lane >> 3), c0 = lane & 7;
            const size_t step = (size_t)8 * p.row_bytes;
            RingPlace ring_at(0);
            for (uint32_t j = 0; ts_work<CL>(p, j, wk); j++) {
                const uint32_t rows = min(kBM, p.m - wk.m0);  // rows past the end: whatever is there, nobody stores their results
                for (uint32_t u = wk.kb0 >> 2; u < (wk.kb1 + 3) >> 2; u++, ring_at.advance(1, p.w_stages)) {
                    const uint32_t sw = ring_at.stage(p.w_stages);
                    if (!ring_at.first_use(p.w_stages) && !warp_wait(&empty_w[sw], ring_at.empty_parity(p.w_stages), lane, abort_flag, p.status)) {
                        asm volatile("cp.async.wait_all;" ::: "memory");
                        goto done;
                    }
                    const uint32_t seg = min(Ge::ub, p.row_bytes - u * Ge::ub) + 6;  // the last unit of a row may not be whole
                    const uint32_t dst = smem_u32(smem + p.w_off) + sw * Ge::stage + first * Ge::rs + c0 * Ge::cp;
                    const uint8_t *src = p.w + (size_t)(wk.m0 + first) * p.row_bytes + (size_t)u * Ge::ub;
                    bool live[(Ge::need + 7) / 8];
#pragma unroll
                    for (uint32_t c = 0; c < (Ge::need + 7) / 8; c++) live[c] = (c * 8 + c0) * Ge::cp < seg;
#pragma unroll
                    for (uint32_t r = 0; r < kBM / 8; r++) {
                        if (first + 8 * r < rows) {
                            const uint8_t *at = reinterpret_cast<const uint8_t *>(reinterpret_cast<uintptr_t>(src) & ~(uintptr_t)(Ge::cp - 1)) + c0 * Ge::cp;
#pragma unroll
                            for (uint32_t c = 0; c < (Ge::need + 7) / 8; c++)
                                if (live[c]) cp_async8(dst + 8 * r * Ge::rs + c * 8 * Ge::cp, at + c * 8 * Ge::cp);
                        }
                        src += step;
                    }
                    cp_async_arrive(&full_w[ring_at.full()]);
                }
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
        }
    } else if (warp == kTsTmaWarp) {
        // ---------------- activation tiles
        pdl_wait();  // x may come from the kernel before
        const uint32_t tile = p.box * (kBK * 2);  // bytes
        uint32_t s = 0, use = 0;
        for (uint32_t j = 0; ts_work<CL>(p, j, wk); j++) {
            for (uint32_t g = wk.kb0 / p.b_kb; g * p.b_kb < wk.kb1; g++, s = s + 1 == p.b_stages ? (use++, 0) : s + 1) {
                if (use > 0 && !warp_poll(&empty_b[s], (use - 1) & 1, abort_flag, p.status)) {
                    const long long t0 = clock64();  // as above
                    while (clock64() - t0 < 100000) {}
                    goto done;
                }
                const uint32_t lo = max(g * p.b_kb, wk.kb0), hi = min((g + 1) * p.b_kb, wk.kb1);
                if (elect_one()) {
                    mbar_expect_tx(&full_b[s], (hi - lo) * tile);
                    for (uint32_t kb = lo; kb < hi; kb++)
                        tma_load_tile(smem + p.b_off + (s * p.b_kb + kb - g * p.b_kb) * tile, &xmap, kb * kBK, wk.n0, &full_b[s]);
                }
                __syncwarp();
            }
        }
    } else if (warp == kTsMmaWarp) {
        // ---------------- MMA issuer, a unit a turn
        const uint32_t tile = p.box * (kBK * 2);
        uint32_t item = 0, it = 0, s_b = 0, use_b = 0;
        for (uint32_t j = 0; ts_work<CL>(p, j, wk); j++, item++) {
            // N of the instruction: the tokens the item really has, in sixteens
            const uint32_t live = min(p.tok, p.n - wk.n0), idesc = instr_desc(F16 ? 0u : 1u, kBM, (live + 15u) & ~15u);
            const uint32_t acc = two_acc ? item & 1 : 0, acc_use = two_acc ? item >> 1 : item, d = tmem_base + acc * 128;
            if (acc_use > 0 && !warp_poll(&acc_empty[acc], (acc_use - 1) & 1, abort_flag, p.status)) goto done;
            tc_fence_after();
            for (uint32_t u = wk.kb0 >> 2; u < (wk.kb1 + 3) >> 2; u++, it++) {
                const uint32_t set = it & 1, hi = min(4 * u + 4, wk.kb1);
                if (!warp_poll(&full_a[set], it >> 1 & 1, abort_flag, p.status)) goto done;
                for (uint32_t kb = max(4 * u, wk.kb0); kb < hi; s_b = s_b + 1 == p.b_stages ? (use_b++, 0) : s_b + 1) {
                    if (!warp_poll(&full_b[s_b], use_b & 1, abort_flag, p.status)) goto done;
                    tc_fence_after();
                    const uint32_t end = min((kb / p.b_kb + 1) * p.b_kb, hi);  // of this stage
                    uint64_t db = smem_desc(smem_u32(smem + p.b_off) + (s_b * p.b_kb + kb % p.b_kb) * tile);
                    // (the loop outside, the elected lane inside: see warp_poll)
#pragma unroll 1
                    for (; kb < end; kb++, db += tile >> 4) {
                        const uint32_t a = tmem_base + kTsACol + set * kTsACols + (kb - 4 * u) * 32;
                        const uint32_t dc = CL ? d + ((kb - wk.kb0) & (chains - 1)) * chain_cols : d;
                        const bool begun = CL ? kb - wk.kb0 >= chains : kb != wk.kb0;
                        if (elect_one()) {
#pragma unroll
                            for (uint32_t k4 = 0; k4 < kBK / 16; k4++)
                                // 16 k: eight columns of A, 32 bytes further along B's swizzled 128-byte row
                                umma_ts(dc, a + k4 * 8, db + k4 * 2, idesc, (begun || k4 != 0) ? 1u : 0u);
                        }
                        __syncwarp();
                    }
                    if (elect_one()) umma_commit(&empty_b[s_b]);
                    __syncwarp();
                }
                if (elect_one()) umma_commit(&empty_a[set]);
                __syncwarp();
            }
            if (elect_one()) umma_commit(&acc_full[acc]);
            __syncwarp();
        }
    } else {
        // ---------------- epilogue: four warps, warp q reads tensor-memory lanes 32q .. 32q + 31
        const uint32_t q = warp & 3;
        uint32_t item = 0;
        pdl_wait();  // the kernel before may still read what is written here
        for (uint32_t j = 0; ts_work<CL>(p, j, wk); j++, item++) {
            const uint32_t n_end = min(p.n, wk.n0 + p.tok), row = wk.m0 + q * 32 + lane;
            const uint32_t acc = two_acc ? item & 1 : 0, acc_use = two_acc ? item >> 1 : item;
            if (!warp_wait(&acc_full[acc], acc_use & 1, lane, abort_flag, p.status)) goto done;
            tc_fence_after();
            // partial tiles hold all 128 rows
            float *part = wk.slot < kTsShare ? p.partial + (size_t)wk.slot * p.nt * kBM + q * 32 + lane : nullptr;
#pragma unroll 1
            for (uint32_t t0 = wk.n0; t0 < n_end; t0 += 32) {
                uint32_t r[32];
                tmem_ld32(tmem_base + ((q * 32) << 16) + acc * 128 + (t0 - wk.n0), r);
                tmem_ld_wait();
                const uint32_t live = min(32u, n_end - t0);
                if (CL) {
                    // Into shared memory, where the rings were: every copy into them has been read by the MMAs that are complete.
                    const uint32_t o = smem_u32(smem + p.b_off) + (t0 - wk.n0) * (kBM * 4) + (q * 32 + lane) * 4;
#pragma unroll
                    for (uint32_t i = 0; i < 32; i++)
                        if (i < live) sts32(o + i * (kBM * 4), r[i]);
#pragma unroll 1
                    for (uint32_t c = 1; c < chains; c++) {  // a thread's own words
                        tmem_ld32(tmem_base + ((q * 32) << 16) + c * chain_cols + (t0 - wk.n0), r);
                        tmem_ld_wait();
#pragma unroll
                        for (uint32_t i = 0; i < 32; i++)
                            if (i < live) sts32(o + i * (kBM * 4), __float_as_uint(__uint_as_float(lds32(o + i * (kBM * 4))) + __uint_as_float(r[i])));
                    }
                } else if (part) {
                    float *o = part + (size_t)(t0 - wk.n0) * kBM;
#pragma unroll
                    for (uint32_t i = 0; i < 32; i++)
                        if (i < live) o[i * kBM] = __uint_as_float(r[i]);
                } else if (row < p.m) {
                    if (p.nout == 0 && p.odt == DT_F32) {
                        float *o = reinterpret_cast<float *>(p.out) + (size_t)t0 * p.m + row;
#pragma unroll
                        for (uint32_t i = 0; i < 32; i++)
                            if (i < live) o[(size_t)i * p.m] = __uint_as_float(r[i]);
                    } else if (p.nout == 0) {
                        __nv_bfloat16 *o = reinterpret_cast<__nv_bfloat16 *>(p.out) + (size_t)t0 * p.m + row;
#pragma unroll
                        for (uint32_t i = 0; i < 32; i++)
                            if (i < live) o[(size_t)i * p.m] = __float2bfloat16_rn(__uint_as_float(r[i]));
                    } else {
                        // row shards: a warp stores 32 consecutive rows of one token (128 bytes) into every
                        // rank's buffer, over NVLink for the other ranks'
#pragma unroll 1
                        for (uint32_t b = 0; b < p.nout; b++) {
                            float *o = reinterpret_cast<float *>(p.outs[b]) + p.out_row0 + row + (size_t)t0 * p.out_ld;
#pragma unroll
                            for (uint32_t i = 0; i < 32; i++)
                                if (i < live) o[(size_t)i * p.out_ld] = __uint_as_float(r[i]);
                        }
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[acc]);
        }
    }
done:
    if constexpr (CL) {
        // Every CTA of the cluster adds up every so many-th token, in the order of k, out of the others' shared memory.
        pdl_wait();  // (the kernel before may still read what is written here)
        __syncwarp();
        cluster_sync();
        ts_work<CL>(p, 0, wk);
        const uint32_t live = min(p.tok, p.n - wk.n0), rank = blockIdx.x % p.cluster;
        for (uint32_t t = rank * (kTsThreads / 32) + warp; t < live; t += p.cluster * (kTsThreads / 32)) {
            const uint32_t at = smem_u32(smem + p.b_off) + t * (kBM * 4) + lane * 16;
            float4 v[8];
#pragma unroll
            for (uint32_t c = 0; c < 8; c++)
                if (c < p.cluster) v[c] = lds_of(at, c);
#pragma unroll
            for (uint32_t c = 1; c < 8; c++)
                if (c < p.cluster) v[0] = make_float4(v[0].x + v[c].x, v[0].y + v[c].y, v[0].z + v[c].z, v[0].w + v[c].w);
            store_rows(p, v[0], wk.m0, wk.n0 + t, lane);
        }
        cluster_sync();  // nobody leaves while its part may still be read
    }
    if (p.epoch && !p.dealt && blockIdx.x == 0 && threadIdx.x == 0) {
        pdl_wait();
        p.epoch[0] += p.epoch_inc;
    }
    tc_fence_before();
    __syncthreads();
    if (warp == kTsMmaWarp) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

template <int TY, bool SK, bool F16, bool CL>
static cudaError_t ts_launch(TsArgs a, const void *x, uint32_t grid, cudaStream_t s, int dev) {
    using Ge = TsGeom<TY, SK>;
    static bool attr_set[64] = {};  // the opt-in is per device
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (!attr_set[dev]) {
        cudaError_t e = cudaFuncSetAttribute(gemm_ts_kernel<TY, SK, F16, CL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTsSmem);
        if (e != cudaSuccess) return e;
        attr_set[dev] = true;
    }
    // Shared memory: barriers, the activations' ring (1024-byte aligned tiles, 16 to 32 KB a stage), the weights' ring, tables.
    // What the activations do not need of it (96 KB, or eight stages) holds weights on their way from HBM.
    a.box = a.tok < ((a.n + 15u) & ~15u) ? a.tok : (a.n + 15u) & ~15u;
    a.b_kb = a.box <= 64 ? 4 : a.box <= 128 ? 2 : 1;
    const uint32_t b_stage = a.b_kb * a.box * kBK * 2, tab = TY == T_IQ2_XXS ? 384 * 4 * kTsTabCopies : 0;
    const uint32_t room = kTsSmem - 1024 /*align*/ - 1024 /*barriers*/ - tab - 16 /*reads past the last row*/;
    uint32_t b_least = 96 * 1024 / b_stage;
    if (b_least > 8) b_least = 8;
    a.w_stages = (room - b_least * b_stage) / Ge::stage;
    if (a.w_stages > kTsMaxW) a.w_stages = kTsMaxW;
    a.b_stages = (room - a.w_stages * Ge::stage) / b_stage;
    if (a.b_stages > kTsMaxB) a.b_stages = kTsMaxB;
    a.b_off = 1024;
    a.w_off = a.b_off + a.b_stages * b_stage;
    a.tab_off = a.w_off + a.w_stages * Ge::stage;
    alignas(64) CUtensorMap xmap, wmap;
    memset(&wmap, 0, sizeof(wmap));
    cudaError_t e = encode_x_map(&xmap, x, a.k, a.n, a.box);
    if (e != cudaSuccess) return e;
    // The weights' tensor map: a row of it is as many rows of the matrix as make a multiple of 16 bytes.
    a.tma_log = 0;
    while (((uint64_t)a.row_bytes << a.tma_log) % 16) a.tma_log++;
    const uint64_t pitch = (uint64_t)a.row_bytes << a.tma_log;
    if (SK && ((uintptr_t)a.w % 16 || a.m % (1u << a.tma_log))) {
        a.tma_log = kTsNoTma;
    } else {
        e = encode_map(&wmap, CU_TENSOR_MAP_DATA_TYPE_UINT32, a.w, pitch / 4, a.m >> a.tma_log, pitch, Ge::rs / 4, kBM >> a.tma_log,
                       CU_TENSOR_MAP_SWIZZLE_NONE);
        if (e != cudaSuccess) return e;
    }
    return launch_pdl(gemm_ts_kernel<TY, SK, F16, CL>, grid, kTsThreads, kTsSmem, s, CL ? a.cluster : 1, xmap, wmap, a);
}
template <int TY, bool SK>
static cudaError_t ts_launch_x(const TsArgs &a, const void *x, int xdt, uint32_t grid, cudaStream_t s, int dev) {
    if constexpr (TY != T_Q4_0)  // (see share_out)
        if (a.cluster > 1) return xdt == DT_F16 ? ts_launch<TY, SK, true, true>(a, x, grid, s, dev) : ts_launch<TY, SK, false, true>(a, x, grid, s, dev);
    return xdt == DT_F16 ? ts_launch<TY, SK, true, false>(a, x, grid, s, dev) : ts_launch<TY, SK, false, false>(a, x, grid, s, dev);
}

}  // namespace tc

const uint32_t *gemm_ts_clusters(int dev) {
    struct Known {
        std::once_flag once;
        uint32_t room[9] = {};
    };
    static Known known[64];
    if (dev < 0 || dev >= 64) return nullptr;
    Known &k = known[dev];
    std::call_once(k.once, [&] {
        auto kernel = tc::gemm_ts_kernel<T_Q4_K, false, true, true>;
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tc::kTsSmem) != cudaSuccess) {
            (void)cudaGetLastError();
            return;
        }
        for (uint32_t c = 2; c <= 8; c++) {
            cudaLaunchAttribute at;
            at.id = cudaLaunchAttributeClusterDimension;
            at.val.clusterDim.x = c;
            at.val.clusterDim.y = at.val.clusterDim.z = 1;
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(c * 256);
            cfg.blockDim = dim3(tc::kTsThreads);
            cfg.dynamicSmemBytes = tc::kTsSmem;
            cfg.attrs = &at;
            cfg.numAttrs = 1;
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, (const void *)kernel, &cfg) != cudaSuccess) {
                (void)cudaGetLastError();
                n = 0;
            }
            k.room[c] = (uint32_t)n;
        }
    });
    return k.room;
}

cudaError_t launch_gemm_ts(const GemmTs &g, cudaStream_t s, int dev) {
    tc::TsArgs a = {};
    a.w = g.w; a.out = g.out; a.status = g.status; a.partial = g.partial;
    a.k = g.k; a.m = g.m; a.n = g.n; a.row_bytes = g.row_bytes;
    a.tok = g.tok; a.groups = (g.n + g.tok - 1) / g.tok; a.items = (g.m + tc::kBM - 1) / tc::kBM * a.groups;
    a.waves = g.waves; a.dealt = g.dealt; a.dealers = g.dealers; a.nt = g.nt;
    a.odt = (uint32_t)g.odt;
    a.cluster = g.cluster;
    a.chains = g.chains;
    a.vec = g.m % 4 == 0 && (g.nout ? (g.out_ld | g.out_row0) % 4 == 0 : (uintptr_t)g.out % (g.odt == DT_F32 ? 16 : 8) == 0);
    for (uint32_t i = 0; i < g.nout; i++) a.vec = a.vec && (uintptr_t)g.outs[i] % 16 == 0;
    a.nout = g.nout; a.out_ld = g.out_ld; a.out_row0 = g.out_row0; a.epoch = g.epoch; a.epoch_inc = g.epoch_inc;
    for (uint32_t i = 0; i < g.nout; i++) a.outs[i] = g.outs[i];
    const uint32_t all = (uint32_t)g.sms, grid = a.cluster > 1 ? a.items * a.cluster : a.waves ? all : a.dealt ? a.dealers : a.items < all ? a.items : all;
    const bool whole = ((uintptr_t)g.w | g.row_bytes) % 16 == 0;  // (units of these four types are multiples of 16 bytes)
    switch (g.ty) {
    case T_Q4_K: return tc::ts_launch_x<T_Q4_K, false>(a, g.x, g.xdt, grid, s, dev);
    case T_Q5_K: return whole ? tc::ts_launch_x<T_Q5_K, false>(a, g.x, g.xdt, grid, s, dev) : tc::ts_launch_x<T_Q5_K, true>(a, g.x, g.xdt, grid, s, dev);
    case T_Q8_0: return whole ? tc::ts_launch_x<T_Q8_0, false>(a, g.x, g.xdt, grid, s, dev) : tc::ts_launch_x<T_Q8_0, true>(a, g.x, g.xdt, grid, s, dev);
    case T_Q4_0: return whole ? tc::ts_launch_x<T_Q4_0, false>(a, g.x, g.xdt, grid, s, dev) : tc::ts_launch_x<T_Q4_0, true>(a, g.x, g.xdt, grid, s, dev);
    case T_IQ4_NL: return whole ? tc::ts_launch_x<T_IQ4_NL, false>(a, g.x, g.xdt, grid, s, dev) : tc::ts_launch_x<T_IQ4_NL, true>(a, g.x, g.xdt, grid, s, dev);
    case T_Q6_K: return tc::ts_launch_x<T_Q6_K, true>(a, g.x, g.xdt, grid, s, dev);
    case T_Q2_0: return tc::ts_launch_x<T_Q2_0, true>(a, g.x, g.xdt, grid, s, dev);
    case T_IQ2_XXS: return tc::ts_launch_x<T_IQ2_XXS, true>(a, g.x, g.xdt, grid, s, dev);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace okf
