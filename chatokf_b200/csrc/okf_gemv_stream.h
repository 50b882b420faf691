// The plan of a streaming matvec (okf_gemv_stream.cu): how its units are dealt to CTAs and warps, what lies where in shared memory,
// and which of the possible splits a launch takes.  Host code, but for the arithmetic by which a CTA finds its share.
#pragma once
#include "okf_gemv_unit.cuh"

namespace okf {

// A warp's ring: `depth` stages of 16 row segments, `cb` units each.  Segments are copied from the 32-byte boundary below them
// (a sector of L2 is fetched once); they lie 16 bytes into their rows of the stage, and up to 14 more where they start between 16-byte
// boundaries.
template <int TY, int MODE> struct StreamGeom {
    static constexpr uint32_t ub = UnitGeom<TY>::bytes;
    static constexpr bool rag = WideMode<MODE>::rag, aligned = ub % 16 == 0 && !rag;
    // Units of a stage: as many as make a segment of some 100 to 300 bytes (Q2_0 2048 -> 6144 twice, one column, two and four units: 4.5
    // and 4.2 us); in several columns' kernels, whose x takes the room, fewer.
    static constexpr uint32_t cb = ub < 68 ? (MODE == M_SEP ? 2 : 1) : ub < 100 ? (MODE == M_SEP ? 4 : 2) : 1;
    static constexpr uint32_t bytes = 16 + (aligned ? cb * ub : (cb * ub + 14 + 15) / 16 * 16);
    // Rows g and g + 1 of a tile on different banks: an odd number of 16 bytes apart for 16- and 4-byte loads; where a quad's
    // 8-byte loads lie side by side, 32 bytes modulo 64.
    static constexpr uint32_t pitch = aligned && MODE != M_SEP ? bytes + (96 - bytes % 64) % 64 : bytes % 32 == 16 ? bytes : bytes + 16;
    static constexpr uint32_t stage = 16 * pitch;
};

struct StreamLayout {
    uint32_t nc, es;      // activation columns, bytes between byte columns of the x panel
    uint32_t clog;        // log2 of the CTAs of a cluster, each with its share of K of the cluster's tiles
    uint32_t depth;       // stages of a warp's ring: 2 to 4
    uint32_t xs_off, info_off, slot_off, part_off, tab_off;  // byte offsets in dynamic shared memory
    uint32_t tab_copies;  // IQ2_XXS: copies of every entry of the look-up tables, side by side
    uint32_t tile_first;                 // of this launch
    uint32_t tiles_each, tiles_more;     // tiles of a cluster; the first tiles_more clusters have one more
    __host__ __device__ void deal(uint32_t first, uint32_t tiles, uint32_t clusters) {
        tile_first = first;
        tiles_each = tiles / clusters;
        tiles_more = tiles % clusters;
    }
    uint32_t unit_inv, unit_inv_more;    // v / units = v * inv >> 31, for CTAs with nunit >> clog units of a row and with one more
    uint32_t nc_inv;                     // v / nc = v * nc_inv >> 16, v < 8192
};

// A CTA's units of its tiles laid end to end; warp w has [border(w), border(w + 1)).
struct StreamSplit {
    uint32_t nun, all, inv;  // units of a tile, of all tiles
    __host__ __device__ __forceinline__ StreamSplit(uint32_t tiles, uint32_t units, uint32_t inv_) : nun(units), all(tiles * units), inv(inv_) {}
    template <uint32_t NW> __host__ __device__ __forceinline__ uint32_t border(uint32_t w) const { return all * w / NW; }
    __host__ __device__ __forceinline__ uint32_t tile(uint32_t v) const { return (uint32_t)((uint64_t)v * inv >> 31); }
};
inline uint32_t stream_inv(uint32_t units) { return (0x80000000u + units - 1) / units; }
// Where tile(), border() and nc_inv are exact.
inline bool stream_exact(uint32_t tiles, uint32_t units, uint32_t n) {
    return (uint64_t)tiles * units * units < 0x80000000ull && (uint64_t)tiles * units * 16 < 0x100000000ull && (uint64_t)tiles * n < 8192;
}

// ---- which split a launch takes ----------------------------------------------------------
// What the device has room for: clusters of 1, 2, 4 and 8 CTAs at one CTA to an SM and at two.  (GPCs do not have a multiple of eight
// SMs, so these are fewer than SMs / size: a grid of 37 clusters of four on 148 SMs takes two waves, twice the time.)
struct StreamRoom {
    uint32_t one[4], two[4];
};
struct StreamPlan {
    bool ok, early;  // early: may start beside its predecessor
    uint32_t warps, ctas, smem;
    uint32_t tiles;  // of a launch: all, or (see stream_launches) the launches of a matrix take that many each, the last one what is left
    float us;  // estimated, of all launches
    StreamLayout L;
};
// (two of 112 KB leave 2 KB of an SM: enough for the small kernels between matvecs, which with 1 KB less take 0.8 us longer each)
constexpr uint32_t stream_budget(uint32_t warps) { return warps == 8 ? 112 * 1024 : 226 * 1024; }

// What a CTA of a grid that is meant to be one to an SM asks for: two of them do not fit one SM.  Left to themselves two end up on one SM and
// none on another where a grid comes while SMs fall free one by one: 197 such launches of all types but IQ2_XXS take 7 % longer when
// launches follow one another, 5 % behind elementwise kernels (Q2_0 2048 -> 2048 and its like, eight layers, 131 -> 124 us; in a graph of
// matvecs alone 1 %, 6 % the other way for grids of exactly as many CTAs as SMs).  IQ2_XXS's CTAs fill 48 KB of tables first, which they can
// do beside their predecessors: alone 5 % slower there and 5 % faster behind elementwise kernels, so without clusters they are left.
constexpr uint32_t kStreamAlone = 116 * 1024;

// Clusters of four and eight at two CTAs to an SM, all the device has room for, need every SM: beside a predecessor that still holds some (a small kernel holds
// registers) clusters that lie across them wait, and what they leave free does not hold a cluster either, so some start when others end, half as long again
// (IQ2_XXS 24320 -> 28385, 4 columns, behind an elementwise kernel 201.7 us, 138.5 when it starts behind it; in a chain of matvecs 131.8 and
// 134.4).  From this estimate on they start when their predecessor is complete: 61 shapes 0.693 of the other kernel's time over three kinds of chain, 0.702
// if all start early, 0.722 if none does; below it the 3 us that an early start hides weigh more (IQ2_XXS 17408 -> 5120, 4 columns, 19.8 and 22.4 in a chain of matvecs).
constexpr float kStreamLate = 27.f;

template <int TY, int MODE>
inline bool stream_layout(uint32_t nunit, uint32_t n, uint32_t clog, uint32_t clusters, uint32_t tiles, uint32_t warps, StreamPlan &p) {
    using S = StreamGeom<TY, MODE>;
    constexpr bool sep = MODE == M_SEP;
    StreamLayout &L = p.L;
    const uint32_t tiles_per = (tiles + clusters - 1) / clusters, units = (nunit + (1u << clog) - 1) >> clog;
    const uint32_t nb = mode_bytes(MODE), ecols = sep ? 2 : n * nb;
    if (!stream_exact(tiles_per, units, n)) return false;
    L.nc = n;
    L.clog = clog;
    L.es = sep ? sep_col_stride(units) : xq_col_stride(units);
    // the deepest ring that leaves room for x and, IQ2_XXS, for tables without bank conflicts; else half the tables
    for (L.tab_copies = TY == T_IQ2_XXS ? 32 : 0;; L.tab_copies = 16) {
        for (L.depth = 4; L.depth >= 2; L.depth--) {
            L.xs_off = (warps * L.depth * S::stage + 127) & ~127u;
            L.info_off = (L.xs_off + ecols * L.es + 15) & ~15u;
            L.slot_off = (L.info_off + (sep ? 256u : units * n * wide_info_words(TY, nb) * 4) + 127) & ~127u;  // (one column: 256 bytes of zeros before it)
            L.part_off = L.slot_off + warps * 2 * n * 64;
            L.tab_off = L.part_off + (clog ? tiles_per * n * 64 : 0);
            p.smem = L.tab_off + 384 * 4 * L.tab_copies;
            if (p.smem <= stream_budget(warps)) break;
        }
        if (L.depth >= 2) break;
        if (L.tab_copies != 32) return false;
    }
    p.warps = warps;
    p.ctas = clusters << clog;
    L.deal(0, tiles, clusters);
    L.unit_inv = stream_inv(nunit >> clog);
    L.unit_inv_more = stream_inv((nunit >> clog) + 1);
    L.nc_inv = 65536 / n + 1;
    return true;
}

// The time of a launch in a chain, us: what it takes whatever its size, a warp's staging of x (column, unit pairs) and a warp's units,
// both at another rate where two CTAs share an SM, and never less than the weights take at what copies in pieces of 16 bytes reach (4.9
// TB/s).  The constants are fits, one up to four columns and one for what is left: to 21 000 and to 44 000 timings, of
// 1080 and 1480 shapes (every type, 1 to 8 columns, rows of 384 to 18432 weights, 300 to 150 000 rows), each in a chain of matvecs, in one
// with an elementwise kernel before every matvec and, in the second fit, in a chain of plain launches, as engines have them all.  The choice made
// with them is 0.9 % slower than the best one at one column (geometric mean over the shapes; at most 16 %), 0.7 to 1.3 % at several.  Against
// okf_gemv.cu's kernel alone 633 other shapes are, in the first and second kind of chain, 1.08 and 1.11 times as fast at one column, 1.18
// and 1.20 at two to four, 1.31 and 1.34 at five to eight, 1.15 to 1.24 where rows end inside a unit; a fifth and a twentieth of
// them at one column, a twentieth of the others, lose more than 2 %.  One CTA to an SM where there is work for two is the faster one in the
// first kind of chain only (Q4_K 2560 -> 2 x 9728, one column, 8.2 and 8.4 us, behind an elementwise kernel 13.5 and 10.4): it leaves room
// for the next matvec's first copies, but what comes behind a small kernel starts its copies late, and two CTAs have more of them in flight.
inline int stream_kind(int mode) { return mode == M_SEP ? 0 : mode == M_W1 ? 1 : mode == M_W2 ? 2 : 3; }
struct StreamUnit {
    float stream[4];  // one column, up to four, up to eight, rows that end inside a unit
    float ring[4];    // the same of okf_gemv.cu's kernel (not asked at five to eight)
};
inline StreamUnit stream_unit_us(int ty) {
    switch (ty) {
    case T_Q4_K: return {{.71f, .75f, .83f, 0.f}, {.44f, .58f, 0.f, 0.f}};
    case T_Q8_0: return {{1.23f, 1.50f, 1.25f, 1.18f}, {.82f, 1.00f, 0.f, .76f}};
    case T_Q6_K: return {{1.40f, 1.61f, 1.39f, 0.f}, {.87f, .80f, 0.f, 0.f}};
    case T_Q5_K: return {{.90f, 1.01f, 1.03f, 0.f}, {.72f, .94f, 0.f, 0.f}};
    case T_Q4_0: return {{.70f, 1.03f, .93f, .96f}, {.34f, .61f, 0.f, .55f}};
    case T_IQ4_NL: return {{1.16f, 1.29f, 1.04f, 1.08f}, {.92f, .70f, 0.f, .97f}};
    case T_Q2_0: return {{.51f, .71f, .70f, .67f}, {.28f, .33f, 0.f, .44f}};
    default: return {{.95f, 1.20f, 1.04f, 0.f}, {.67f, .89f, 0.f, 0.f}};
    }
}
inline float quad_max(float a, float b) { return sqrtf(sqrtf(a * a * a * a + b * b * b * b)); }  // the larger one, rounded off
inline float stream_us(int ty, int mode, uint32_t nunit, uint32_t n, uint32_t tiles, uint32_t clog, uint32_t clusters, uint32_t warps, bool shared, float floor_us) {
    const int kind = stream_kind(mode);
    constexpr float one[2][4] = {{1.3f, 2.65f, 3.05f, 4.2f}, {1.95f, 3.3f, 3.4f, 4.1f}};  // up to four columns, the others; by cluster size, one CTA to an SM
    constexpr float two[4][4] = {{2.5f, 3.8f, 7.8f, 8.1f}, {3.2f, 4.5f, 8.5f, 8.9f}, {2.8f, 4.85f, 9.f, 10.f}, {1.65f, 3.7f, 7.85f, 9.f}};
    constexpr float wide[4] = {4.35f, 6.25f, 6.5f, 8.05f};  // sixteen warps
    constexpr float stage[4] = {.59f, .62f, .35f, .51f}, stage_two[4] = {1.3f, .66f, 1.1f, 1.75f}, unit_two[4] = {.71f, .78f, 1.42f, 1.37f};
    const uint32_t units = (nunit + (1u << clog) - 1) >> clog, per = (tiles + clusters - 1) / clusters * units;
    const float busy = stream_unit_us(ty).stream[kind] * (float)((per + warps - 1) / warps) * (shared ? unit_two[kind] : 1.f) +
                       stage[kind] * (float)((units * n + warps - 1) / warps) * (shared ? stage_two[kind] : 1.f);
    return (warps == 16 ? wide[clog] : shared ? two[kind][clog] : one[kind / 2][clog]) + quad_max(busy, floor_us);
}
// The same of okf_gemv.cu's kernel, whose CTAs share their tiles' units between eight warps; `ctas` and `clog` as it would take them.
// It is asked where it may be the better one: at one column, where its bulk copies of whole rows reach 6.1 TB/s (Q4_K 5120 -> 65536 33.6
// us, 39.2 here), and at up to four where an SM gets four tiles and more, to which x is staged once.  Five to eight columns are better off here
// (Q4_K 2560 -> 9728 twice, 17.4 -> 12.3 us, 9728 -> 2560 19.7 -> 10.8; of 240 shapes with rows of one to six units none is slower, 0.76 of the time on average).
inline float ring_us(int ty, int mode, uint32_t nunit, uint32_t n, uint32_t tiles, uint32_t ctas, uint32_t clog, uint32_t sms) {
    const int kind = stream_kind(mode);
    if (kind == 2 || (kind != 0 && tiles < 4 * sms)) return 1e30f;
    constexpr float fixed[4] = {3.26f, 3.12f, 0.f, 4.65f}, pair_us[2] = {.9f, .77f}, shared_x[2] = {1.32f, 1.65f}, cluster_us[2] = {3.07f, 3.5f};
    const bool shared = ctas > (kind < 2 ? sms : sms + sms / 4);  // (up to a quarter more CTAs than SMs hardly slow each other down where rows end inside a unit)
    const uint32_t clusters = ctas >> clog, units = (nunit + (1u << clog) - 1) >> clog;
    const float busy = (stream_unit_us(ty).ring[kind] * (float)((tiles + clusters - 1) / clusters * units) + pair_us[kind / 2] * (float)(units * n)) / 8.f * (shared ? shared_x[kind / 2] : 1.f);
    const uint32_t ub = ty == T_Q8_0 ? 272 : ty == T_Q6_K ? 210 : ty == T_Q5_K ? 176 : ty == T_Q2_0 ? 68 : ty == T_IQ2_XXS ? 66 : 144;
    float us = fixed[kind] + (shared ? 1.45f : 0.f) + (clog ? cluster_us[kind / 2] : 0.f) + quad_max(busy, (float)nunit * (float)tiles * (16.f * (float)ub / 6.1e6f));
    // One column: where this is too high by 1300 shapes in three kinds of chain.  A tile to a CTA and two CTAs on some SMs only (73 shapes that would all be on the
    // other kernel: 0.960 of this one's time on average and 22 slower by more than 3 % in plain chains, 25 in graphs; with the factor 0.953, 5 and 6; Q8_0 2304 -> 2729 3.7 us,
    // 4.7 there); clusters (31: 0.918 -> 0.915); two CTAs on every SM, three types (101: 0.944 -> 0.947, slower by more than 3 % 18 -> 8; Q6_K 3072 -> 27634 17.7, 21.9 there).
    if (kind == 0 && ctas > sms) us *= ctas < 2 * sms ? .7f : clog || ty == T_Q8_0 ? .85f : ty == T_Q6_K || ty == T_IQ4_NL ? .9f : 1.f;
    return tiles < 12 * sms ? us : kind == 3 && n == 1 ? .85f * us : .93f * us;  // (with so many tiles the fit favours the other kernel: ragged Q4_0 2336 -> 63677
                                                                                 // 27.5 us here, 32.5 there)
}

template <int TY, int MODE>
inline StreamPlan stream_search(uint32_t nunit, uint32_t n, uint32_t tiles, const StreamRoom &room) {
    StreamPlan best = {};
    const float floor_us = (float)nunit * (float)tiles * (16.f * UnitGeom<TY>::bytes / 4.9e6f);
    for (uint32_t clog = 0; clog < 4 && (clog == 0 || nunit >= 2u << clog); clog++) {
        for (uint32_t v = 0; v < (MODE == M_W2 ? 3 : 2); v++) {
            const uint32_t warps = v == 2 ? 16 : 8, limit = v == 1 ? room.two[clog] : room.one[clog], clusters = tiles < limit ? tiles : limit;
            // Two CTAs to an SM from five columns on and at rows that end inside a unit only where they fill nine tenths of the places: fewer
            // are spread unevenly, two on one SM and one on another (the fit without this rule chooses 1 % worse).
            const bool fills = MODE == M_SEP || MODE == M_W1 ? tiles > room.one[clog] : (clusters << clog) * 10 >= room.two[0] * 9;
            if (clusters == 0 || (v == 1 && !fills)) continue;
            StreamPlan p = {};
            if (!stream_layout<TY, MODE>(nunit, n, clog, clusters, tiles, warps, p)) continue;
            // There is an SM for every CTA.  (Asked of the number of CTAs, 34 to 37 clusters of four and 16 to 18 of eight went out as grids with an SM a CTA, of which 33 and 15
            // fit at once: 25 shapes took 1.8 times as long.)
            const bool alone = clusters <= room.one[clog];
            p.us = stream_us(TY, MODE, nunit, n, tiles, clog, clusters, warps, warps == 16 || !alone, floor_us);
            p.ok = true;
            p.tiles = tiles;
            p.early = clog < 2 || alone || p.us < kStreamLate;
            if (warps == 8 && alone && p.smem < kStreamAlone && (TY != T_IQ2_XXS || clog)) p.smem = kStreamAlone;
            if (!best.ok || p.us < best.us) best = p;
        }
    }
    return best;
}

// Where no split fits (tall matrices of long rows at several columns: in clusters, which x needs, a CTA keeps the sums of all its cluster's tiles) the tiles are
// dealt to several launches, each with room for its own: as few as fit, or up to twice as many if they are estimated to be better.  Such matrices went to the other
// kernel, which stages x anew for every few tiles: 82 shapes of all types, 2 to 8 columns, take 0.55 of its time (IQ2_XXS 23040 -> 64269, 8 columns, 802 -> 292 us, Q8_0
// 5376 -> 80310, 8, 127 -> 110; that kernel in clusters, with all of x, 697 and 341).  Not rows of Q8_0 and Q4_0 that end inside a unit, whose x of three and four bytes
// leaves rings of two stages (Q8_0 7904 -> 59634, 5 columns, 245 and 294).
template <int TY, int MODE>
inline StreamPlan stream_launches(uint32_t nunit, uint32_t n, uint32_t tiles, const StreamRoom &room) {
    StreamPlan best = stream_search<TY, MODE>(nunit, n, tiles, room);
    if (best.ok || (WideMode<MODE>::rag && (TY == T_Q8_0 || TY == T_Q4_0))) return best;
    for (uint32_t parts = 2, most = 64; parts <= most && parts <= tiles; parts++) {
        StreamPlan p = stream_search<TY, MODE>(nunit, n, (tiles + parts - 1) / parts, room);
        if (!p.ok) continue;
        if (!best.ok) most = 2 * parts;
        p.us *= (float)parts;
        if (!best.ok || p.us < best.us) best = p;
    }
    return best;
}

// The search costs the host as much as a launch and an engine asks for the same few shapes on every token: a thread keeps
// the plans it found last.
template <int TY, int MODE>
inline const StreamPlan &stream_plan(uint32_t nunit, uint32_t n, uint32_t tiles, const StreamRoom &room, int dev) {
    struct Entry {
        uint32_t nunit, n, tiles;
        int dev;
        StreamPlan p;
    };
    constexpr uint32_t kEntries = 16;
    static thread_local Entry kept[kEntries];  // (tiles = 0: none yet)
    Entry &e = kept[((nunit * 31 + n) * 31 + tiles) * 2654435761u >> 28];
    static_assert(kEntries == 16, "four bits of the hash");
    if (e.nunit != nunit || e.n != n || e.tiles != tiles || e.dev != dev) e = {nunit, n, tiles, dev, stream_launches<TY, MODE>(nunit, n, tiles, room)};
    return e.p;
}

// How many launches of this kernel took the matvec; 0: it is not one for it (or does not fit), and nothing was launched.
struct GemvArgs;
int launch_gemv_stream(int ty, int mode, const GemvArgs &a, int xdt, cudaStream_t s, int sms, int dev, float other_us, cudaError_t &e);

}  // namespace okf
