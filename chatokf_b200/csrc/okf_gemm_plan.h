// Which plan a prefill matmul takes.  Host code, but for the rule by which its kernels find their own share of dealt work.
#pragma once
#include <stddef.h>
#include <stdint.h>

#include "okf_blocks.cuh"

namespace okf {

// How a matmul is laid over the SMs.  A work item is a 128-row slab against some tokens over all of K.  Full waves of items
// run whole, one item per CTA and wave.  What is left after them, or a matmul of less than a wave, either runs whole too, on
// part of the SMs, or is dealt out: its k (k-blocks here, units of 256 in okf_gemm_ts.cu) laid end to end is cut into one run per
// CTA, pieces of items leave as fp32 partial tiles, and a second kernel sums them.  The plan with the smallest estimated time wins.
// The estimate, measured on B200: 0.86 us per k-block on an item of 512 tokens (Q8_0 0.92, Q6_K 1.1), which exposes 3 us of
// epilogue, and what ts_kblock says on one of fewer.  Dealing is counted as 6 us and partial tiles at 8 TB/s, mostly
// through L2.  (Timed both ways, in chains of calls, on 112 shapes whose plan depends on it, 9 to 3800 tokens, all types: counted as 2.5 us the
// plan taken is 8.5 % slower than the better one on average, as 5 us 2.8 %, as 6 us 1.7 %, as 7.5 us 0.8 %, as 10 us 1.8 %.  A call that is
// waited for, as the host-buffer operator's are, pays less for the second kernel: Q4_0 2304 -> 2071, 11 tokens, host to host 37.2 us dealt,
// 39.1 whole, Q2_0 2304 -> 5376, 14 tokens, 50.4 and 51.9; with 7.5 us counted they would run whole.
// Dealt and whole, us: Q8_0 1024 -> 8570, 11 tokens, 10.0 and 4.8; Q4_0 2560 -> 9728, 77 tokens, 15.4 and 13.3; Q5_K the same 16.6 and
// 14.8; Q5_K 5376 -> 5888, 147 tokens, 22.6 and 27.9; 9728 -> 2560, 77 tokens, 17.6 and 42.  4096 tokens 17408 -> 5120: 320 items of two
// blocks are 2.16 waves; three whole waves took 760 us, two and 24 dealt items 590.)
// Sums in tensor memory cut off where fp32 would round, so a whole item is further from the exact sum than a dealt one with its shorter
// chains: 1.2e-6 of the result after 1024 k, 1.9e-5 after 17408 (a rounding of an operand to fp16 2e-4).
struct GemmPlan {
    uint32_t tok;    // tokens per item of the kernel with weights in tensor memory, 0: the other one
    uint32_t nacc;   // token blocks per item
    uint32_t waves, dealt, dealers, nt;  // see tc::Args
    uint32_t cluster;  // CTAs of a cluster that share an item along K, 0: none; tok != 0 and all items at once
    uint32_t chains;   // shared items: accumulators that take their k-blocks in turn
    size_t floats;   // of partial tiles
};

namespace tc {

constexpr uint32_t kBM = 128;  // weight rows per CTA tile (UMMA M)
constexpr uint32_t kBN = 256;  // tokens per accumulator (UMMA N)
constexpr uint32_t kBK = 64;   // k per stage: 64 x 2 bytes = one 128-byte swizzle row

// Dealing: CTA c takes k-blocks [total * c / ctas, total * (c + 1) / ctas) of the dealt items laid end to
// end.  The CTA that takes k-block x (total * ctas stays below 2^32):
__host__ __device__ __forceinline__ uint32_t dealt_to(uint32_t x, uint32_t total, uint32_t ctas) { return ((x + 1) * ctas - 1) / total; }

}  // namespace tc

// The better of running `slabs` x `groups` items of `tok` tokens whole and of dealing the last wave out, into `best` if it
// beats `best_t`.  An item is `steps` of k long; t_step: seconds for one; t_item: what an item adds; `least`: steps a CTA takes at least.
inline void lay_out(GemmPlan plan, uint32_t slabs, uint32_t steps, uint32_t n, uint32_t tok, double t_step, double t_item, uint32_t least, uint32_t all,
                    size_t max_floats, GemmPlan &best, double &best_t) {
    const uint32_t base = slabs * ((n + tok - 1) / tok);
    const double whole = ((base + all - 1) / all) * (steps * t_step + t_item);
    if (whole < best_t) { best_t = whole; best = plan; }
    // the items of the last, part-filled wave (of the only one) dealt out by steps
    const uint32_t waves = base / all, dealt = base % all, nt = n < tok ? n : tok;
    if (dealt == 0) return;
    const uint64_t total = (uint64_t)dealt * steps;
    if (total * (all + 1) >= 0xFFFFFFFFull) return;
    uint32_t ctas = total / least < all ? (uint32_t)(total / least) : all;
    if (ctas <= dealt) return;
    uint32_t parts = 1;
    for (uint32_t i = 0; i < dealt; i++) {
        const uint32_t c = tc::dealt_to((i + 1) * steps - 1, (uint32_t)total, ctas) - tc::dealt_to(i * steps, (uint32_t)total, ctas) + 1;
        if (c > parts) parts = c;
    }
    const size_t part = (size_t)dealt * nt * tc::kBM;  // floats
    if (parts * part > max_floats) {
        // as many equal parts of every item as there is room for (Q4_K 9728 -> 2560, 512 tokens, in 16 MiB: on 40
        // of the SMs 71 us with fp16 and 358 with fp32 activations, in three parts on 120 of them 35 and 196)
        parts = (uint32_t)(max_floats / part);
        if (parts > steps / least) parts = steps / least;
        if (parts > all / dealt) parts = all / dealt;
        if (parts < 2) return;
        ctas = dealt * parts;
    }
    const double moved = 2.0 * (dealt + ctas) * nt * tc::kBM * 4;
    const double t = waves * (steps * t_step + t_item) + ((total + ctas - 1) / ctas) * t_step + 6e-6 + moved / 8e12;
    if (t < best_t) {
        best_t = t;
        best = plan;
        best.waves = waves; best.dealt = dealt; best.dealers = ctas; best.nt = nt; best.floats = parts * part;
    }
}
// The same items, each by a cluster of CTAs that cut its K among them and add up in each other's shared memory: no second kernel and no working
// memory, but all items have to be there at once.  `room`: how many clusters of a size fit the device.  The exchange is counted as 2 us and 5 ns a
// token, 1.5 us more against items that run whole: of 84 shapes (9 to 1020 tokens, all types) that were timed with and without, the plan taken
// is 0.8 % slower than the better one on average (never counting the 1.5 us; 5 % if they are counted against dealt items too).  Dealt or whole, and shared, us:
// Q5_K 9728 -> 2560, 77 tokens, 19.8 and 17.6; Q2_0 6144 -> 2048, 512 tokens, 22.6 and 19.5; Q4_K 4608 -> 403, 256 tokens, 12.1 and 8.6; IQ4_NL
// 3840 -> 1307, 13 tokens, 11.9 and 6.1; whole items that stay whole: Q4_K 1792 -> 1840, 158 tokens, 7.9 and 8.4.
// Clusters of three and five, whose CTAs share a pair of SMs with another cluster's, do not take the last sixteenth of the room, and those of two that would take
// whole items' place not all of it: while SMs fall free one by one, behind a kernel of some other grid (the one that converts x, an elementwise one),
// the last clusters find no SMs side by side and start in a second wave (43 to 45 clusters of three, 80 shapes: 17 % slower than without behind an elementwise
// kernel, up to 1.8 times, Q4_K 6912 -> 526, 794 tokens of fp32, 23.7 and 30.4; 39 to 42 of them 4 % faster.  Clusters of five 2 % slower and 8 % faster;
// all the room taken by 49 grids of four, six, seven and eight CTAs 8 to 15 % faster).
// Whole items of fewer than eight units are shared by three CTAs or more where a seventh of the room is left: 32 shapes 8 to 17 % faster; by two CTAs, or
// with less room left, 54 shapes 1 % faster to 8 % slower (Q6_K 1536 -> 2774, 259 tokens, 10.4 and 12.5).
// Q4_0 does not share, though it would gain as the others do (4096 -> 1500, 34 tokens, 13.6 us instead of 9.0; 120 shapes of 9 to 1024 tokens take 0.916 of the time in plain
// chains): test_gpu_tile_dealing.py and test_gpu_tile_memory.py hold that its calls deal, by the number of their kernels.
// Sums in tensor memory are cut off where fp32 would round, so a chain's error grows with its length.  `base`: units of a chain of the plan without
// clusters; where an item's parts are longer, their k-blocks go to two or four accumulators in turn (there is room for
// them up to 128 and 64 tokens), which are added up at the end, and where that is not enough the split is not taken.  500 shapes of fp16 operands, rms
// errors against 64 bits: the 303 that share are 0.74 of the plans without clusters on average, at most 1.04 times (chains a quarter longer
// let through: 0.84 and 1.35).  One more accumulator costs 0.3 us at 77 tokens; 260 shapes are 0.5 % slower on average than with longer chains.
inline void share_out(GemmPlan plan, uint32_t slabs, uint32_t units, uint32_t n, uint32_t tok, double t_unit, double t_item, double base, const uint32_t *room,
                      bool whole, GemmPlan &best, double &best_t) {
    const uint32_t items = slabs * ((n + tok - 1) / tok);
    for (uint32_t c = 2; c <= 8; c++) {
        const uint32_t places = c == 3 || c == 5 ? room[c] * 15 / 16 : c == 2 && whole && room[c] ? room[c] - 1 : room[c];
        if (items > places || units < 2 * c) continue;
        if (whole && units < 8 && (c == 2 || items > room[c] * 6 / 7)) continue;
        const uint32_t most = tok <= 64 ? 4 : tok <= 128 ? 2 : 1;
        const double part = (units + c - 1) / c;
        uint32_t chains = 1;
        while (chains < most && part > chains * base) chains *= 2;
        if (part > chains * base) continue;
        const double t = (units + c - 1) / c * t_unit + t_item + 2e-6 + (n < tok ? n : tok) * 5e-9;
        if (t + (whole && !best.cluster ? 1.5e-6 : 0) < best_t) { best_t = t; best = plan; best.cluster = c; best.chains = chains; }
    }
}
// 16-bit activations: seconds per k-block of an item of `tok` tokens on the kernel with weights in tensor memory.  Up to
// some 100 tokens the unpacking sets the pace, above that it grows with the tokens (5120 -> 17408, 80 k-blocks an SM: 22.7 to 29.4 us
// at 64 tokens, Q4_K 29.5 at 128, 56 at 256).
inline double ts_kblock(int ty, uint32_t tok) {
    const double unpack = ty == T_Q8_0 ? 0.29e-6 : ty == T_Q6_K ? 0.335e-6 : ty == T_IQ2_XXS || ty == T_IQ4_NL ? 0.3e-6 : ty == T_Q5_K ? 0.26e-6 : 0.23e-6;
    const double stream = 0.17e-6 + 1.1e-9 * tok;
    return unpack > stream ? unpack : stream;
}
// Items may be of any number of tokens (fewer than 256 where that gives every SM one: Q2_0 2048 -> 6144, 512 tokens, in 144 items of
// 176 tokens 16 us, in 96 of 256 17, in 48 of 512 20).
// `room`: see share_out; null: no clusters.
inline GemmPlan gemm_tc_search(int ty, uint32_t k, uint32_t m, uint32_t n, int xdt, int sms, size_t max_floats, const uint32_t *room = nullptr) {
    const uint32_t slabs = (m + tc::kBM - 1) / tc::kBM, kblocks = k / tc::kBK, all = (uint32_t)sms;
    GemmPlan best = {}, plan = {};
    double best_t = 1e30;
    if (xdt == DT_F32) {
        // fp32 activations that the tile converts itself, by one group of warps while another unpacks:
        // 0.9 us, from some 80 tokens on what the conversion takes, 2.3 us at 256
        plan.nacc = 1;
        lay_out(plan, slabs, kblocks, n, tc::kBN, n > 80 ? 0.3e-6 + 7.8e-9 * (n < tc::kBN ? n : tc::kBN) : 0.9e-6, 0, 4, all, max_floats, best, best_t);
        return best;
    }
    if (n > tc::kBN) {
        plan.nacc = 2;
        lay_out(plan, slabs, kblocks, n, 2 * tc::kBN, ty == T_Q6_K ? 1.1e-6 : ty == T_Q8_0 ? 0.92e-6 : 0.86e-6, 3e-6, 4, all, max_floats, best, best_t);
        plan.nacc = 0;
    }
    const uint32_t least = (n + tc::kBN - 1) / tc::kBN;
    for (uint32_t blocks = least; blocks <= least + 8; blocks++) {
        plan.tok = ((n + blocks - 1) / blocks + 15) / 16 * 16;
        lay_out(plan, slabs, (kblocks + 3) / 4, n, plan.tok, 4 * ts_kblock(ty, plan.tok), plan.tok > 128 ? 2.5e-6 : 1e-6, 1, all, max_floats, best, best_t);
        if (plan.tok <= 32) break;
    }
    if (!room || ty == T_Q4_0) return best;
    const uint32_t units = (kblocks + 3) / 4;
    const double run = best.dealt && !best.waves ? (double)best.dealt * units / best.dealers : units, base = run < 1 ? 1 : run;
    const bool whole = !best.dealt;
    for (uint32_t blocks = least; blocks <= least + 8; blocks++) {
        const uint32_t tok = ((n + blocks - 1) / blocks + 15) / 16 * 16;
        plan = {};
        plan.tok = tok;
        share_out(plan, slabs, units, n, tok, 4 * ts_kblock(ty, tok), tok > 128 ? 2.5e-6 : 1e-6, base, room, whole, best, best_t);
        if (tok <= 32) break;
    }
    return best;
}

// The search costs the host up to 4 us (512 tokens: nine widths of items, each with a loop over the dealt ones) and an engine
// asks for the same few shapes in every layer, so each thread keeps the plans it found last.  (Searched anew, and twice, in every
// call: Q2_0 2048 -> 6144, 512 tokens, took the host 11.5 us beside 16 on the GPU.)
inline GemmPlan gemm_tc_plan(int ty, uint32_t k, uint32_t m, uint32_t n, int xdt, int sms, size_t max_floats, const uint32_t *room = nullptr) {
    struct Entry {
        int ty, xdt, sms;
        uint32_t k, m, n;
        size_t max_floats;
        const uint32_t *room;  // (one array a device, never changed)
        bool used;
        GemmPlan plan;
    };
    constexpr uint32_t kEntries = 64;
    static thread_local Entry cache[kEntries];
    uint32_t h = (((uint32_t)ty * 31 + k) * 31 + m) * 31 + n;
    h = (h * 4 + (uint32_t)xdt) * 2 + (max_floats != 0);
    Entry &e = cache[(h * 2654435761u) >> 26];
    static_assert(kEntries == 64, "six bits of the hash");
    if (!(e.used && e.ty == ty && e.xdt == xdt && e.sms == sms && e.k == k && e.m == m && e.n == n && e.max_floats == max_floats && e.room == room))
        e = {ty, xdt, sms, k, m, n, max_floats, room, true, gemm_tc_search(ty, k, m, n, xdt, sms, max_floats, room)};
    return e.plan;
}

}  // namespace okf
