// The plan of a matvec on gemv_kernel (okf_gemv.cu): how tiles are dealt to CTAs, what a stage of the ring holds and what lies where in
// shared memory, and what such a launch is estimated to take beside okf_gemv_stream.cu's.  Host code.
#pragma once
#include "okf_gemv_stream.h"

namespace okf {

struct GemvLayout {
    uint32_t mode;         // 0: stage = tps x 16 whole rows, 1: stage = 8 whole rows, 2: stage = 16 row segments
    uint32_t rs;           // bytes between rows inside a stage
    uint32_t stage_bytes;
    uint32_t nstage;       // ring depth
    uint32_t tps;          // tiles per stage (mode 0 only, else 1)
    uint32_t ragged;       // mode 2: row segments do not start on 16-byte boundaries
    uint32_t group;        // tiles summed per barrier
    uint32_t nc;           // activation columns of this pass
    uint32_t nc_inv;       // i / nc = i * nc_inv >> 16 for the few hundred (tile, column) pairs of a group
    uint32_t es;           // bytes between columns of the x panel
    uint32_t panel;        // k-chunks whose slice of x is staged together
    uint32_t clog;         // log2 of the CTAs of a cluster, each with its share of K of the cluster's tiles (0: no clusters)
    uint32_t xs_off, info_off, red_off, tab_off, part_off;  // byte offsets in dynamic shared memory
    uint32_t tab_copies;   // IQ2_XXS: copies of every codebook entry, side by side (a power of two)
    uint32_t smem_bytes;
};

constexpr uint32_t kBarBytes = 512;   // barriers and the abort flag, then 256 bytes of zeros at kZeroOff
constexpr uint32_t kMaxStages = 8;

// Shared-memory plan.  Two CTAs share an SM (this launch's and the next one's,
// already prefetching), so each gets at most 112 KB.  (A launch with many tiles
// per CTA gains nothing from taking the SM for itself with a deeper ring: at
// that size the kernel is bound by instruction issue, not by bytes in flight.)
//
// Ring stages.  A bulk copy costs the copy engine about 50 ns however small it
// is, and a stage hand-over costs the consumers a few hundred cycles, so stages
// are large (20 - 46 KB) and filled by as few copies as possible: when whole rows
// fit, a stage is up to four tiles (or half a tile) of consecutive rows and one
// contiguous copy -- which also makes the 2-byte-aligned layouts copyable, since
// 8 rows always start on a 16-byte boundary -- otherwise rows are cut into
// segments of at least 1 KB, one copy per row.  `tiles_per_cta` is the most tiles
// any CTA of the launch gets.
constexpr uint32_t kSharedBudget = 112 * 1024;  // two of them leave 2 KB of an SM: enough for the small kernels between matvecs

inline uint32_t unit_bytes(int ty) {
    return (ty == T_Q4_K || ty == T_Q4_0 || ty == T_IQ4_NL) ? 144 : ty == T_Q8_0 ? 272 : ty == T_Q2_0 ? 68 : ty == T_Q6_K ? 210 : ty == T_Q5_K ? 176 : 66;
}
inline bool gemv_layout_with(int ty, uint32_t row_bytes, uint32_t nunit, uint32_t n, int mode, uint32_t csize, uint32_t tiles_per_cta,
                             uint32_t tab_copies, uint32_t budget, GemvArgs &a, GemvLayout &L) {
    const uint32_t ub = unit_bytes(ty);
    const bool sep = mode == M_SEP;
    L.nc = n;
    L.nc_inv = 65536 / n + 1;
    L.clog = csize == 8 ? 3 : csize == 4 ? 2 : csize == 2 ? 1 : 0;
    const uint32_t nb = mode_bytes(mode);
    const bool rag = nb > 2;
    const uint32_t ecols = sep ? 2 : n * nb;  // byte columns of the x panel
    const uint32_t units = (nunit + csize - 1) / csize;   // the most a CTA of a cluster takes
    const uint32_t per_tile = kGemvWarps * 16 * L.nc * 4;
    const uint32_t part_bytes = csize > 1 ? tiles_per_cta * 16 * L.nc * 4 : 0;
    const uint32_t tab_bytes = ty == T_IQ2_XXS ? 384 * 4 * tab_copies : 0;
    L.tab_copies = tab_copies;
    const uint32_t stage_cap = 46 * 1024;
    // per unit: SEP 320 bytes per byte column, records included; WIDE 256 per byte column and the columns' records
    const uint32_t xunit = sep ? kSepUnit : kXqUnit, info_unit = sep ? 0 : n * wide_info_words(ty, nb) * 4;
    GemvArgs fb_a = a;
    GemvLayout fb_L = L;
    bool have_fallback = false;
    // One candidate; true when it is taken.  `red`: bytes of partial sums, a group of tiles.
    auto consider_with = [&](uint32_t kind, uint32_t tps, uint32_t nchunk, uint32_t red) {
        L.group = red / per_tile;
        if (L.group < tps) L.group = tps;
        if (L.group > tiles_per_cta) L.group = tiles_per_cta;
        const uint32_t red_bytes = L.group * per_tile;
        L.mode = kind;
        L.tps = tps;
        L.ragged = 0;
        uint32_t cb = units, rs = row_bytes, stage;
        if (kind == 0) {
            stage = (tps * 16 * rs + 15) & ~15u;
        } else if (kind == 1) {
            stage = (8 * rs + 15) & ~15u;
        } else {
            cb = (units + nchunk - 1) / nchunk;
            if ((units + cb - 1) / cb != nchunk) return false;
            const uint32_t seg = cb * ub;
            L.ragged = (row_bytes % 16 || ub % 16) ? 1 : 0;
            // Q4_K reads its blocks with 16-byte loads, and its rows are always aligned
            if (L.ragged && !rag && ty != T_IQ2_XXS && ty != T_Q2_0 && ty != T_Q6_K) return false;
            rs = L.ragged ? ((seg + 15 + 15) & ~15u) : seg;  // room for the skipped bytes and the round-up
            if (rs % 32 != 16) rs += 16;                      // rows g and g + 1 on different banks
            stage = 16 * rs;
        }
        if (stage > stage_cap) return false;
        a.nchunk = nchunk;
        a.cb = cb;
        L.rs = rs;
        L.stage_bytes = stage;
        const uint32_t per_chunk = ecols * cb * xunit + cb * info_unit;  // x and what goes with it
        const uint32_t small = kBarBytes + red_bytes + part_bytes + tab_bytes + 64 + 128 + ecols * 128;
        const uint32_t min_stages = kind == 1 ? 4 : 2;
        if (small + min_stages * stage + per_chunk > budget) return false;
        uint32_t nstage, panel;
        if (small + min_stages * stage + nchunk * per_chunk <= budget) {
            panel = nchunk;  // all of x resident, the rest goes to the ring
            nstage = (budget - small - nchunk * per_chunk) / stage;
        } else {
            nstage = min_stages;
            panel = (budget - small - min_stages * stage) / per_chunk;
        }
        // no deeper than the steps a CTA takes
        const uint32_t steps = ((tiles_per_cta + tps - 1) / tps) * nchunk * (kind == 1 ? 2 : 1);
        if (nstage > steps) nstage = steps < min_stages ? min_stages : steps;
        if (nstage > kMaxStages) nstage = kMaxStages;
        if (kind == 1) nstage &= ~1u;  // a tile takes two stages
        L.nstage = nstage;
        L.panel = panel;
        L.es = sep ? sep_col_stride(panel * cb) : xq_col_stride(panel * cb);
        L.xs_off = (kBarBytes + nstage * stage + 127) & ~127u;  // the bank arithmetic of the panel counts from 128
        L.info_off = (L.xs_off + ecols * L.es + 15) & ~15u;
        L.red_off = (L.info_off + panel * cb * info_unit + 15) & ~15u;
        L.tab_off = (L.red_off + red_bytes + 15) & ~15u;
        L.part_off = L.tab_off + tab_bytes;
        L.smem_bytes = L.part_off + part_bytes;
        if (L.smem_bytes > budget) return false;
        // A plan that keeps all of x resident stages it once per launch; one that does
        // not stages a slice per k-chunk, every time with all warps waiting.
        if (panel == nchunk) return true;
        if (!have_fallback) { fb_a = a; fb_L = L; have_fallback = true; }
        return false;
    };
    // with fewer tiles to a group where that makes room for the plan
    auto consider = [&](uint32_t kind, uint32_t tps, uint32_t nchunk) {
        for (uint32_t red = sep ? 8192 : 16384; red >= (sep ? 8192u : 4096u); red /= 2)
            if (consider_with(kind, tps, nchunk, red)) return true;
        return false;
    };
    // Candidate plans, best first: whole tiles, several per stage while they are small and the CTA
    // still gets two steps, half tiles, then one copy per row of ever shorter segments.
    // Contiguous rows cannot be padded: when the row size is a multiple of 64 bytes the rows a
    // warp reads together sit on the same banks, and per-row copies with a padded stride come
    // first.  Plans with all of x resident are preferred as long as their row segments stay
    // above 1 KB.
    const bool same_banks = row_bytes % 64 == 0;
    if (csize == 1) {
        if (same_banks && consider(2, 1, 1)) return true;
        for (uint32_t tps = 4; tps >= 1; tps--)
            if (tps == 1 || (tps * 16 * row_bytes <= stage_cap && tps * 2 <= tiles_per_cta))
                if (consider(0, tps, 1)) return true;
        if (consider(1, 1, 1)) return true;
    }
    for (uint32_t nchunk = 1; nchunk <= units; nchunk++) {
        if (!(same_banks && csize == 1 && nchunk == 1) && consider(2, 1, nchunk)) return true;
        if (have_fallback && (units / (nchunk + 1)) * ub < 1024) break;
    }
    if (have_fallback) { a = fb_a; L = fb_L; }
    return have_fallback;
}

// IQ2_XXS: as many side-by-side copies of the look-up tables as leave room for a plan that
// keeps all of x resident (32 copies make every look-up free of bank conflicts).
inline bool gemv_layout_search(int ty, uint32_t row_bytes, uint32_t nunit, uint32_t n, int mode, uint32_t csize, uint32_t tiles_per_cta, GemvArgs &a,
                               GemvLayout &L) {
    // (Tried for several columns of long rows, whose panel of x does not fit beside the ring in
    // half an SM's shared memory: taking the SM alone with the whole panel resident.  Slower:
    // the next kernel can then not prefetch under this one.)
    if (ty != T_IQ2_XXS) return gemv_layout_with(ty, row_bytes, nunit, n, mode, csize, tiles_per_cta, 1, kSharedBudget, a, L);
    GemvArgs fa = a;
    GemvLayout fl = L;
    bool have = false;
    for (uint32_t copies = 32; copies >= 1; copies /= 2) {
        GemvArgs ta = a;
        GemvLayout tl = L;
        if (!gemv_layout_with(ty, row_bytes, nunit, n, mode, csize, tiles_per_cta, copies, kSharedBudget, ta, tl)) continue;
        if (tl.panel == ta.nchunk) { a = ta; L = tl; return true; }
        if (!have) { fa = ta; fl = tl; have = true; }
    }
    if (have) { a = fa; L = fl; }
    return have;
}

// The search costs the host about as much as a launch and an engine asks for the same few
// shapes on every token, so each thread keeps the plans it found last.
inline bool gemv_layout(int ty, uint32_t row_bytes, uint32_t nunit, uint32_t n, int mode, uint32_t csize, uint32_t tiles_per_cta, GemvArgs &a,
                        GemvLayout &L) {
    struct Entry {
        int ty, mode;
        uint32_t row_bytes, nunit, n, csize, tiles_per_cta, cb, nchunk;
        bool used, ok;
        GemvLayout L;
    };
    constexpr uint32_t kEntries = 64;
    static thread_local Entry cache[kEntries];
    uint32_t h = ((uint32_t)ty * 31 + row_bytes) * 31 + n;
    h = ((h * 31 + tiles_per_cta) * 8 + csize) * 8 + (uint32_t)mode;
    Entry &e = cache[(h * 2654435761u) >> 26];
    static_assert(kEntries == 64, "six bits of the hash");
    if (!(e.used && e.ty == ty && e.mode == mode && e.row_bytes == row_bytes && e.nunit == nunit && e.n == n && e.csize == csize && e.tiles_per_cta == tiles_per_cta)) {
        GemvArgs t = {};
        e = {ty, mode, row_bytes, nunit, n, csize, tiles_per_cta, 0, 0, true, false, {}};
        e.ok = gemv_layout_search(ty, row_bytes, nunit, n, mode, csize, tiles_per_cta, t, e.L);
        e.cb = t.cb;
        e.nchunk = t.nchunk;
    }
    if (!e.ok) return false;
    a.cb = e.cb;
    a.nchunk = e.nchunk;
    L = e.L;
    return true;
}

// CTAs of a launch: one per SM, each with its share of the tiles, with two exceptions.
// When there are only a few more tiles than SMs (160 on 148) two tiles in a row on a dozen SMs would
// set the launch's time, and one CTA per tile is used instead; an SM has room for two of them side
// by side, and they do not slow each other down much (a CTA alone issues on a third of the cycles).
// (One column only: with several columns two CTAs on an SM, each staging its slices of x at
// barriers, were 16 % slower than two tiles in a row.)
// Where an SM has enough to do, two CTAs share it: eight warps wait for one another's instructions on two
// thirds of the cycles, sixteen fill them; against that stand a second panel of x and the lost room for
// the next launch's first copies.  One column: from eight tiles or 144 KB of blocks per SM on, IQ2_XXS,
// which works longest on a byte, counted one and a half times (Q4_K 2560 -> 65536 22.3 -> 18.5 us, Q8_0
// 4096 -> 5120, two tiles per SM, 9.4 -> 8.0; Q4_K 2560 -> 14000, 136 KB, 6.8 -> 7.2), and from 80 KB on
// where that is at most three tiles, which one CTA would take one after another on some SMs (192 to
// 320 tiles: Q8_0 4096 -> 4096 6.7 -> 5.2, Q4_K 12288 -> 3072 11.4 -> 8.7, 5120 -> 5120 6.7 -> 6.1; below, Q4_K
// 4096 -> 4096, 64 KB, 4.15 -> 4.35; not for the two types with a look-up per weight, whose warps hardly
// wait: IQ2_XXS 6144 -> 6144 9.6 -> 10.5, IQ4_NL 10.1 -> 11.3).  Several columns (up to four, and row shards; five to eight are okf_gemv_stream.cu's else, and
// the figures of eight are this kernel's, before there was that one), with more work per tile: from three tiles on (Q4_K 5120 -> 17357, 4 columns, 27.6 -> 20.0 us, 8 columns 35 -> 29;
// 512 tiles, which were left to one CTA per SM: Q5_K 17408 -> 8192, 3 columns, 56.9 -> 40.6 us, Q4_K 20480 -> 8192, 4 columns, 55.6 -> 53.8 us, Q4_K 8192 -> 8192, 8
// columns, 35.6 -> 37.6; the two-bit types, with little to wait for, from four on: IQ2_XXS 8192 -> 8192, 5 columns, 23.6 us, from three 27.5).
inline bool two_bit(int ty) { return ty == T_IQ2_XXS || ty == T_Q2_0; }
inline bool two_ctas(int ty, uint32_t row_bytes, uint32_t tiles, int sms, bool sep) {
    if (!sep) return tiles >= (two_bit(ty) ? 4u : 3u) * (uint32_t)sms;
    const uint64_t raw = (uint64_t)tiles * 16 * row_bytes, bytes = ty == T_IQ2_XXS ? raw + raw / 2 : raw;
    const bool few = tiles <= 3u * (uint32_t)sms && ty != T_IQ2_XXS && ty != T_IQ4_NL;
    return tiles >= 8u * (uint32_t)sms || bytes >= (few ? 81920ull : 147456ull) * (uint32_t)sms;
}
inline uint32_t gemv_ctas(int ty, uint32_t row_bytes, uint32_t tiles, int sms, bool sep) {
    const uint32_t n = (uint32_t)sms;
    if (tiles <= n) return tiles;
    if (two_ctas(ty, row_bytes, tiles, sms, sep)) return tiles < 2 * n ? tiles : 2 * n;
    return sep && tiles <= n + n / 4 ? tiles : n;
}

// Grid and shared-memory plan of a launch.  At one column clusters of CTAs share a tile along K where that lets every CTA keep its part of x
// in shared memory or, for IQ2_XXS, all 32 copies of its tables: the smallest cluster that does.  Where x fits anyway clusters
// cost time (Q4_K 9728 -> 2560 7.1 -> 7.9), except for long rows with some more tiles than two to an SM: tiles halved between two CTAs
// spread evenly over the chip, whole ones leave most CTAs one and a few of them two (Q4_K 17408 -> 5120 21.3 -> 16.9 us, Q8_0 32.7 ->
// 24.6; Q8_0 5120 -> 5120, 20 units of 272 bytes, 8.8 -> 9.5, Q4_K 9216 -> 5120, 36 of 144, 10.3 -> 10.8; the line lies somewhere
// between these points).  Several columns of rows that would need a cluster are okf_gemv_stream.cu's, in as many launches as that takes (rows of
// Q8_0 and Q4_0 that end inside a unit come here: 7904 -> 59634, 5 columns, 258 us in clusters, 245 without); row-shard launches have duties by CTA
// number and take none.
inline bool gemv_plan(int ty, uint32_t row_bytes, uint32_t nunit, uint32_t n, int mode, uint32_t tiles, int sms, bool gather, GemvArgs &a,
                      GemvLayout &L, uint32_t &ctas) {
    const uint32_t all = gemv_ctas(ty, row_bytes, tiles, sms, mode == M_SEP), n2 = 2u * (uint32_t)sms;
    const bool halves = mode == M_SEP && tiles > n2 && tiles <= n2 + n2 / 2 && (row_bytes >= 6144 || nunit >= 40) && !gather;
    for (uint32_t cs = halves ? 2 : 1; cs <= 8 && !((gather || mode != M_SEP) && cs > 1) && cs * 4 <= nunit; cs *= 2) {
        const uint32_t limit = (two_ctas(ty, row_bytes, tiles, sms, mode == M_SEP) ? 2 : 1) * (uint32_t)sms / cs;
        const uint32_t clusters = cs == 1 ? all : tiles < limit ? tiles : limit;
        if (!gemv_layout(ty, row_bytes, nunit, n, mode, cs, (tiles + clusters - 1) / clusters, a, L)) continue;
        // (both rules for IQ2_XXS hold at the trunk's sizes they were set for, 5120 and 17408; where between them each starts
        // to pay was not measured)
        const bool last = ty == T_IQ2_XXS && cs == 2;  // shorter segments of its 66-byte units cost more than a resident x gains
        if (!last && (L.panel < a.nchunk || (mode == M_SEP && ty == T_IQ2_XXS && nunit >= 48 && L.tab_copies < 32))) continue;
        ctas = clusters * cs;
        return true;
    }
    ctas = all;
    return gemv_layout(ty, row_bytes, nunit, n, mode, 1, (tiles + all - 1) / all, a, L);
}

// How `n` columns are taken: the mode of the next pass and its columns.
inline int gemv_mode(uint32_t k, int xdt, uint32_t n, uint32_t &take) {
    if (k % 256) {
        take = n < 4 ? n : 4;
        return xdt == DT_F32 ? M_R4 : M_R3;
    }
    take = n;
    return n == 1 ? M_SEP : n <= 4 ? M_W1 : M_W2;
}

// What the launch would take here, a time without end where that is not asked.
inline float ring_estimate(int ty, int mode, const GemvArgs &a, int sms) {
    if (ring_us(ty, mode, a.nunit, a.n, a.tiles, 1, 0, (uint32_t)sms) >= 1e30f) return 1e30f;
    GemvArgs t = a;
    GemvLayout L;
    uint32_t ctas;
    if (!gemv_plan(ty, a.row_bytes, a.nunit, a.n, mode, a.tiles, sms, false, t, L, ctas)) return 1e30f;
    // Several columns: x resident is not enough, copies have to be on their way as well (Q8_0 17408 -> 8192, 2 columns, with less than 44 KB
    // of ring 88.4 us, shared by two CTAs 42.2).  Asked of every plan: 27 shapes of two to four columns whose ring holds a CTA's whole share, or of two-bit
    // types, that the estimates alone would leave here take 0.62 to 0.98 of this kernel's time on the other one.
    if (mode != M_SEP && (L.panel < t.nchunk || L.nstage * L.stage_bytes < 44 * 1024)) return 1e30f;
    return ring_us(ty, mode, a.nunit, a.n, a.tiles, ctas, L.clog, (uint32_t)sms);
}

}  // namespace okf
