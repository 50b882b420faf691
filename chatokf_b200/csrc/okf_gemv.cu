// Decode matvec kernels (1..8 activation columns) for every block type.  Replaces the reference's kq_gemv_impl / kq_gemm_nb_impl / q2_0_gemv
// families (LLM/metal/Kernels.metal:26-109, :1572-1753), with okf_gemv_stream.cu, which takes most launches of several columns, short
// rows and K cut between CTAs; here go large matrices at one to four columns, and row shards.  See okf_gemv_mma.cuh
// for the data path and the MMA operand layout.
//
// Work split.  A tile is 16 consecutive output rows; a unit is 256 consecutive
// k of a row (one Q4_K / IQ2_XXS super-block, eight Q8_0 blocks, two Q2_0
// blocks).  A CTA owns a contiguous range of tiles.  The producer thread brings
// tiles into a ring of shared-memory stages; when whole rows fit, a stage is a
// few tiles (or half a tile) of consecutive rows and one contiguous bulk copy,
// otherwise rows are cut into k-chunks and a stage takes one segment per row.
// The eight consumer warps deal the units of a stage among themselves, add what
// they computed into their own slots of a partial-sum buffer, and after a group
// of tiles the slots are summed in warp order and stored, so results do not
// depend on timing.
//
// Activations.  Each 256-wide unit of a column of x is reduced to 16-bit integers
// with one fp32 scale, x ~ xs * q, |q| <= 32512 (round to nearest; the step is
// 2^-15 of the unit's largest magnitude), and q is split into two signed bytes,
// q = 256 * hi + lo.  Every kernel here works on these values, so one column
// gives the same result whatever the batch width.
//
// Integer tensor cores.  Weights go into the MMA as the bytes they are stored as
// (nibbles and 2-bit codes after one AND, Q8_0 untouched, IQ2_XXS and IQ4_NL as
// looked up), x as the hi / lo bytes, mma.sync m16n8k32 with s32 accumulators:
// the sums are exact integers; scales, mins and biases are applied afterwards.
//   One column ("SEP"): MMA column g stands for (quarter g / 2 of the unit, byte
// g % 2 of x).  Thread c of a quad owns the k of quarter c and feeds x only into
// that quarter's columns, so the accumulator a thread reads back is the sum over
// exactly the 64 k whose block scales it decoded.
//   Several columns ("WIDE"): see okf_gemv_wide.cuh.
#include <cooperative_groups.h>

#include "okf_gemv_ring.h"
#include "okf_kernels.h"

namespace okf {

// ---- the kernel ---------------------------------------------------------------------
// Position in the ring of stages; the producer and the consumers step through it
// in the same order, so both keep one of these.
struct RingPos {
    uint32_t s = 0, use = 0;  // slot, and how many times the ring wrapped
    __device__ __forceinline__ void next(uint32_t nstage) {
        if (++s == nstage) { s = 0; use++; }
    }
};

// XDT: element type of x.  CL: launched in clusters.  (Both were run-time once: the code a launch does not
// need costs instruction-cache misses that every CTA's staging waits for; Q2_0 2048 -> 2048 3.12 us, so 2.8,
// Q6_K 2560 -> 151936 90.5, so 85.8.)
template <int TY, int MODE, int XDT, bool CL>
__global__ void __launch_bounds__(kGemvThreadsMax, 2) gemv_kernel(GemvArgs p, GemvLayout L, GemvGather G) {
    constexpr uint32_t UB = UnitGeom<TY>::bytes;
    constexpr bool SEP = MODE == M_SEP;
    using W = WideMode<MODE>;
    extern __shared__ __align__(128) uint8_t smem[];
    uint64_t *full = reinterpret_cast<uint64_t *>(smem);
    uint64_t *empty = full + kMaxStages;
    volatile int *abort_flag = reinterpret_cast<volatile int *>(empty + kMaxStages);
    uint8_t *stages = smem + kBarBytes;
    float *part = reinterpret_cast<float *>(smem + L.part_off);  // clusters: [tile][column][16], this CTA's share of K
    float *red = reinterpret_cast<float *>(smem + L.red_off);  // [tile in group][warp][16][nc]
    const uint32_t smem32 = smem_u32(smem);

    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
    // the cluster's tiles and this CTA's units of them
    const uint32_t clog = CL ? L.clog : 0;
    const uint32_t rank = blockIdx.x & ((1u << clog) - 1), cid = blockIdx.x >> clog, ncl = gridDim.x >> clog;
    const uint32_t t0 = (uint32_t)((uint64_t)p.tiles * cid / ncl);
    const uint32_t t1 = (uint32_t)((uint64_t)p.tiles * (cid + 1) / ncl);
    const uint32_t ntl = t1 - t0;
    const uint32_t ubeg = p.nunit * rank >> clog, nun = (p.nunit * (rank + 1) >> clog) - ubeg;
    const uint32_t spt = L.mode == 1 ? 2 : 1;  // stages per step (two half-tiles in mode 1)

    pdl_launch_dependents();
    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < L.nstage; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], kGemvWarps);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x < 64) reinterpret_cast<uint32_t *>(smem + kZeroOff)[threadIdx.x] = 0u;
    if constexpr (TY == T_IQ2_XXS) {
        // the look-up tables, every entry `tab_copies` times side by side (see Iq2Tab)
        uint32_t *tw = reinterpret_cast<uint32_t *>(smem + L.tab_off);
        const uint32_t sh = 31 - __clz(L.tab_copies);
        for (uint32_t i = threadIdx.x; i < 384u; i += blockDim.x) {
            const uint32_t v = i < 256 ? iq2_code_selectors(g_iq2xxs_grid[i]) : iq2_sign_selectors(i - 256);
            for (uint32_t k = 0; k < L.tab_copies; k++) tw[(i << sh) + ((k + threadIdx.x) & (L.tab_copies - 1))] = v;
        }
    }
    __syncthreads();

    // Steps are visited in the same order by the producer and the consumers: group
    // by group, inside a group k-chunk by k-chunk, inside that `tps` tiles at a time.
    if (warp == kGemvWarps + 1) {
        // ---- present in row-shard launches only: announce the exchange of the launch before
        if (lane == 0 && blockIdx.x == 0 && G.sig_nranks) {
            pdl_wait();
            gather_signal(G.sig_arrivals, G.sig_nranks);
        }
        return;
    }
    if (warp == kGemvWarps) {
        // ---- producer: weights do not depend on the previous kernel, so it does not wait for it.
        // One thread waits and counts; copies of whole rows are its own, those of row segments are
        // issued by sixteen lanes, one row each (a bulk copy takes its thread some 50 ns).
        if (L.mode != 2 && lane != 0) return;
        const uint32_t all = L.mode != 2 ? 1u : 0xffffffffu;  // the lanes that are left
        RingPos rp;
        uint32_t issued = 0;
        for (uint32_t gb = 0; gb < ntl; gb += L.group) {
            const uint32_t gn = min(L.group, ntl - gb);
            for (uint32_t j = 0; j < p.nchunk; j++) {
                const uint32_t u0 = j * p.cb, nu = nun > u0 ? min(p.cb, nun - u0) : 0u;
                for (uint32_t tl = gb, tn; tl < gb + gn; tl += tn) {
                    const GemvSeg sg = gemv_segment(p, t0 + tl);
                    tn = min(min(L.tps, gb + gn - tl), sg.tile1 - (t0 + tl));  // a step stays inside one matrix
                    for (uint32_t half = 0; half < spt; half++, issued++) {
                        bool ok = true;
                        if (rp.use > 0 && lane == 0)
                            ok = mbar_wait_relaxed(&empty[rp.s], (rp.use - 1) & 1, abort_flag, p.status, kStatusEmptyTimeout);
                        if (!__shfl_sync(all, ok, 0)) {
                            if (lane != 0) return;
                            // giving up: let the copies already issued land before the CTA goes away
                            const uint32_t first = issued > L.nstage ? issued - L.nstage : 0;
                            for (uint32_t d = first; d < issued; d++) {
                                bool landed = false;
                                for (uint32_t i = 0; i < kSpinLimit && !landed; i++)
                                    landed = mbar_try_wait(&full[d % L.nstage], (d / L.nstage) & 1);
                            }
                            return;
                        }
                        const uint32_t row0 = (t0 + tl - sg.tile0) * 16 + half * 8;
                        uint8_t *dst = stages + (size_t)rp.s * L.stage_bytes;
                        if (L.mode != 2) {
                            // whole rows: one copy; the byte count is rounded up to 16, which may
                            // read a few bytes past the last row (weight buffers are padded)
                            const uint32_t want = L.mode == 1 ? 8u : 16u * tn;
                            const uint32_t nrows = row0 < sg.m ? min(want, sg.m - row0) : 0u;
                            const uint32_t bytes = (nrows * p.row_bytes + 15u) & ~15u;
                            if (lane == 0) {
                                mbar_expect_tx(&full[rp.s], bytes);
                                if (bytes) bulk_g2s(dst, sg.w + (size_t)row0 * p.row_bytes, bytes, &full[rp.s]);
                            }
                        } else {
                            // one copy per row segment.  A segment may start anywhere (2-byte
                            // aligned layouts): the copy starts at the 16-byte boundary below it
                            // and the consumers skip the same few bytes.
                            const uint32_t seg = nu * UB;
                            const size_t src = (size_t)min(row0 + (lane & 15), sg.m - 1) * p.row_bytes + (size_t)(ubeg + u0) * UB;
                            const uint32_t skew = (uint32_t)(src & 15), bytes = seg ? (skew + seg + 15u) & ~15u : 0u;
                            const uint32_t total = __reduce_add_sync(0xffffffffu, lane < 16 ? bytes : 0u);
                            if (lane == 0) mbar_expect_tx(&full[rp.s], total);
                            __syncwarp();
                            if (lane < 16 && bytes) bulk_g2s(dst + (size_t)lane * L.rs, sg.w + (src - skew), bytes, &full[rp.s]);
                        }
                        rp.next(L.nstage);
                    }
                }
            }
        }
        return;
    }

    // ---- consumers
    const uint32_t tid = threadIdx.x;  // 0 .. kConsumers - 1
    // A wait that gives up marks the warp dead; a dead warp skips further waits but
    // keeps walking the loops, so the barriers among the consumer warps still match.
    bool alive = true;
    // Every lane asks for itself: what the barrier hands over is seen by the threads that waited on it, and a shuffle from
    // one that did orders no memory (a __syncwarp behind the shuffle does, and costs 1 % of a decode pass; this costs nothing).
    // `seen`: the stage was complete when the lane looked ahead during the step before.  The lanes vote when they wait; Q5_K at one column,
    // where registers are short, when they look (a bit a lane kept until then spills: 4864 -> 30814 26.3 us, with the vote at the
    // wait 27.2, as it was with one lane asking 26.5; for the other types the vote at the wait is the faster by up to 3 %).
    constexpr bool kVoteEarly = TY == T_Q5_K && SEP;
    auto wait_full = [&](uint32_t s, uint32_t use, bool seen) {
        if (alive && !(kVoteEarly ? seen : __all_sync(0xffffffffu, seen)))
            alive = __all_sync(0xffffffffu, mbar_wait(&full[s], use & 1, abort_flag, p.status, kStatusFullTimeout));
    };
    // has the stage at ring position `q` landed?  (asked before a step's arithmetic about the next
    // step's stages, so that the answer is there when the step is over)
    auto peek_full = [&](const RingPos &q) {
        const bool ok = mbar_test_wait(&full[q.s], q.use & 1);
        return kVoteEarly ? __all_sync(0xffffffffu, ok) : ok;
    };
    auto consumer_sync = [&]() { named_bar_sync(1, kConsumers); };

    const uint32_t stages32 = smem32 + kBarBytes;
    Iq2Tab tab = {0, 0, 0};
    if constexpr (TY == T_IQ2_XXS) {
        tab.stride = L.tab_copies * 4;
        tab.code = smem32 + L.tab_off + (lane & (L.tab_copies - 1)) * 4;
        tab.sign = tab.code + 256 * tab.stride;
    }
    // One column: what this thread feeds into column g of the MMA's B operand, byte column g % 2 of x,
    // and only in the lanes of quarter g / 2.  Lanes that feed nothing read zeros (stride 0) instead of
    // predicating every load; their zeros sit on a bank group that the two lanes carrying data in
    // the same 8-lane phase do not touch.
    const SepConst KC = sep_const<TY>(c);
    const bool sep_active = (g >> 1) == c;
    const uint32_t xbase32 = sep_active ? smem32 + L.xs_off + (g & 1) * L.es + c * kSepQuarter
                                        : smem32 + kZeroOff + ((5 * (g >> 1) + 1) & 7) * 16;
    const uint32_t xstride32 = sep_active ? kSepUnit : 0u;
    const uint32_t rec32 = smem32 + L.xs_off + c * kSepQuarter + 64;  // this quarter's record of unit 0
    const uint32_t red32 = smem32 + L.red_off + (warp * 16 + g + 8 * (c & 1)) * 4;  // this thread's slot of tile 0
    // Several columns: the byte column of the panel this thread feeds per set (columns that stand for
    // nothing read column 0; their sums are dropped), the records of this thread's own columns, and
    // those behind the offsets' byte columns (Q4_K, Q5_K: eight sums, Q6_K: sixteen, per plane).
    constexpr uint32_t kInfo = wide_info_words(TY, W::nb) * 4, kPlane = TY == T_Q6_K ? 16 : 8;
    const uint32_t info32 = smem32 + L.info_off;
    uint32_t wx32[W::sets], wi32[W::vals], ws32[W::vals], ws_lo = 0;
    if constexpr (!SEP) {
#pragma unroll
        for (int i = 0; i < W::sets; i++) {
            const uint32_t j = (W::rag ? 0 : 4 * i) + (g >> 1), b = W::rag ? min(2u * i + (g & 1), W::nb - 1u) : g & 1;
            wx32[i] = smem32 + L.xs_off + (j < p.n ? j * W::nb + b : 0u) * L.es + c * 64;
        }
#pragma unroll
        for (int i = 0; i < W::vals; i++) {
            const uint32_t own = 4 * i + c, fed = 4 * i + (g >> 1);
            wi32[i] = info32 + (own < p.n ? own : 0u) * kInfo;
            const uint32_t word = TY == T_Q6_K ? c : c & 1;
            ws32[i] = info32 + (fed < p.n ? fed : 0u) * kInfo + 4 + (g & 1) * kPlane + 4 * word;  // s2 or s1
            ws_lo = (2 - (g & 1)) * kPlane;                                                        // on to s0
        }
    }
    RingPos rp;
    uint32_t rot = 0;  // the deal of units to warps rotates from step to step
    bool seen_a = false, seen_b = false;
    // Everything up to here, and clearing the first group's partial sums, needs nothing from
    // the kernel before this one.
    for (uint32_t i = tid; i < min(L.group, ntl) * kGemvWarps * 16 * L.nc; i += kConsumers) red[i] = 0.f;
    pdl_wait();  // activations come from the previous kernel; outputs may still be read by it
    if (G.wait_arrivals) {
        // x may hold, or derive from, rows other GPUs stored during the exchange launched
        // before this one: it has to be complete on this GPU before anybody reads x.  The
        // weights of this launch are already streaming in meanwhile.
        if (tid == 0) gather_wait(G.wait_arrivals, G.wait_epoch, p.status);
        named_bar_sync(1, kConsumers);
    }
    const void *x = dep_ptr(reinterpret_cast<const uint8_t *>(p.x));
    for (uint32_t gb = 0; gb < ntl; gb += L.group) {
        const uint32_t gn = min(L.group, ntl - gb);
        if (gb > 0)
            for (uint32_t i = tid; i < gn * kGemvWarps * 16 * L.nc; i += kConsumers) red[i] = 0.f;
        for (uint32_t j0 = 0; j0 < p.nchunk; j0 += L.panel) {
            const uint32_t j1 = min(j0 + L.panel, p.nchunk);
            const uint32_t pu0 = j0 * p.cb, pnu = nun > pu0 ? min(j1 * p.cb, nun) - pu0 : 0u;
            if (gb == 0 || L.panel < p.nchunk) {
                // the previous panel is still being read until every warp gets here
                if (gb > 0 || j0 > 0) consumer_sync();
                if constexpr (SEP) stage_x_bytes<TY, XDT>(smem32 + L.xs_off, L.es, x, ubeg + pu0, pnu, tid);
                else stage_x_wide<TY, MODE, XDT>(smem32 + L.xs_off, L.es, smem32 + L.info_off, x, p.k, L.nc, ubeg + pu0, pnu, tid);
            }
            consumer_sync();
            for (uint32_t j = j0; j < j1; j++) {
                const uint32_t u0 = j * p.cb, nu = nun > u0 ? min(p.cb, nun - u0) : 0u;
                const uint32_t pu = u0 - pu0;  // first unit of the chunk inside the panel
                // in whole-row stages a row holds every unit; in segment stages only this chunk's
                const uint32_t ubase = L.mode == 2 ? 0 : u0;
                for (uint32_t tl = gb, tn; tl < gb + gn; tl += tn) {
                    const GemvSeg sg = gemv_segment(p, t0 + tl);
                    tn = min(min(L.tps, gb + gn - tl), sg.tile1 - (t0 + tl));
                    const uint32_t sA = rp.s;
                    wait_full(rp.s, rp.use, seen_a);
                    rp.next(L.nstage);
                    const uint32_t sB = rp.s;
                    if (spt == 2) {
                        wait_full(rp.s, rp.use, seen_b);
                        rp.next(L.nstage);
                    }
                    {   // look ahead at the next step's stage(s)
                        RingPos q = rp;
                        seen_a = peek_full(q);
                        q.next(L.nstage);
                        seen_b = spt == 2 && peek_full(q);
                    }
                    // the step's first tile: rows 0 .. 7 and 8 .. 15; what the copies fetched below the
                    // start of a row's segment is skipped
                    const uint32_t top = stages32 + sA * L.stage_bytes;
                    const uint32_t low = L.mode == 1 ? stages32 + sB * L.stage_bytes : top + 8 * L.rs;
                    uint32_t ra = top + g * L.rs, wdelta = low - top;  // row g; to row g + 8
                    if (L.mode == 2 && L.ragged) {
                        auto skew = [&](uint32_t row) {
                            return (uint32_t)((size_t)min((t0 + tl - sg.tile0) * 16 + row, sg.m - 1) * p.row_bytes + (size_t)(ubeg + u0) * UB) & 15u;
                        };
                        const uint32_t s0 = skew(g);
                        ra += s0;
                        wdelta += skew(g + 8) - s0;
                    }
                    const uint32_t tile_bytes = 16 * L.rs;
                    // Integer instructions run at half the rate of the others on this part and the
                    // unit bodies are full of them, so a warp takes a run of consecutive units of the
                    // step's tn * nu (unit v being unit v % nu of tile v / nu): the loop over a run
                    // within one tile is a counter and a few addresses moved by constants, and the
                    // sums are put away once per run.  The warps that get one unit more than the
                    // others rotate from step to step.
                    const uint32_t total = tn * nu;
                    const uint32_t wr = warp >= rot ? warp - rot : warp + kGemvWarps - rot;
                    const uint32_t share = total / kGemvWarps, extra = total % kGemvWarps;
                    rot = (rot + extra) % kGemvWarps;
                    uint32_t left = share + (wr < extra ? 1u : 0u);
                    uint32_t ti = 0, u = wr * share + min(wr, extra);
                    while (u >= nu && ti + 1 < tn) { u -= nu; ti++; }
                    if constexpr (SEP) {
                        uint32_t wa = ra + ti * tile_bytes + (ubase + u) * UB;
                        uint32_t xa = xbase32 + (pu + u) * xstride32;
                        uint32_t ia = rec32 + (pu + u) * kSepUnit;
                        uint32_t da = red32 + (tl - gb + ti) * (kGemvWarps * 16 * 4);
                        while (left) {
                            const uint32_t run = min(left, nu - u);  // the rest of this tile, or of the share
                            left -= run;
                            float acc[2] = {0.f, 0.f};
#pragma unroll 1
                            for (uint32_t i = run; i; i--) {
                                const uint4 q0 = lds128(xa), q1 = lds128(xa + 16), q2 = lds128(xa + 32), q3 = lds128(xa + 48);
                                const uint32_t xf[16] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w,
                                                         q2.x, q2.y, q2.z, q2.w, q3.x, q3.y, q3.z, q3.w};
                                const uint4 xi = lds128(ia);
                                const uint4 xj = TY == T_Q6_K ? lds128(ia + L.es) : make_uint4(0u, 0u, 0u, 0u);
                                unit_sep<TY>(wa, wa + wdelta, KC, tab, xf, xi, xj, acc);
                                wa += UB;
                                xa += xstride32;
                                ia += kSepUnit;
                            }
                            // each thread of a quad covered another quarter: add them up and put the
                            // sums into the warp's slot of the tile
#pragma unroll
                            for (int e = 0; e < 2; e++) {
                                acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], 1);
                                acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], 2);
                            }
                            if (c < 2) sts32(da, __float_as_uint(__uint_as_float(lds32(da)) + (c ? acc[1] : acc[0])));
                            // on to the first unit of the next tile
                            u = 0;
                            wa += tile_bytes - nu * UB;
                            xa -= nu * xstride32;
                            ia -= nu * kSepUnit;
                            da += kGemvWarps * 16 * 4;
                        }
                    } else {
                        constexpr int NV = W::vals;
                        uint32_t wa = ra + ti * tile_bytes + (ubase + u) * UB;
                        while (left) {
                            const uint32_t run = min(left, nu - u);
                            left -= run;
                            uint32_t xoff = (pu + u) * kXqUnit, ioff = (pu + u) * L.nc * kInfo;
                            uint32_t blocks = p.k / 32 - (ubeg + u0 + u) * 8;  // left in the row
                            float acc[NV][2];
#pragma unroll
                            for (int i = 0; i < NV; i++) acc[i][0] = acc[i][1] = 0.f;
#pragma unroll 1
                            for (uint32_t i = run; i; i--) {
                                WideX<TY, MODE> X;
#pragma unroll
                                for (int r = 0; r < W::sets; r++)
#pragma unroll
                                    for (int q = 0; q < 4; q++) {
                                        const uint4 v = lds128(wx32[r] + xoff + ((q * 16) ^ ((c >> 1) * 16)));
                                        X.f[r][4 * q] = v.x; X.f[r][4 * q + 1] = v.y; X.f[r][4 * q + 2] = v.z; X.f[r][4 * q + 3] = v.w;
                                    }
#pragma unroll
                                for (int r = 0; r < NV; r++) {
                                    X.scale[r] = __uint_as_float(lds32(wi32[r] + ioff));
                                    if constexpr (TY == T_Q4_K || TY == T_Q5_K || TY == T_Q6_K) {
                                        X.sum[r][0] = lds32(ws32[r] + ioff);
                                        X.sum[r][1] = lds32(ws32[r] + ioff + ws_lo);
                                    } else if constexpr (TY == T_Q2_0) {
#pragma unroll
                                        for (int e = 0; e < 2 * W::nb; e++) X.sum[r][e] = lds32(wi32[r] + ioff + 4 + 4 * e);
                                    }
                                }
                                unit_wide<TY, MODE>(wa, wa + wdelta, c, X, tab, blocks, acc);
                                wa += UB;
                                xoff += kXqUnit;
                                ioff += L.nc * kInfo;
                                if constexpr (W::rag) blocks -= 8;
                            }
                            // into this warp's own slots of the tile's partial sums
                            float *dst = red + ((size_t)(tl - gb + ti) * kGemvWarps + warp) * 16 * L.nc;
#pragma unroll
                            for (int i = 0; i < NV; i++)
                                if (4 * i + c < L.nc) {
                                    dst[g * L.nc + 4 * i + c] += acc[i][0];
                                    dst[(g + 8) * L.nc + 4 * i + c] += acc[i][1];
                                }
                            // on to the first unit of the next tile
                            wa += tile_bytes - nu * UB;
                            u = 0;
                            ti++;
                        }
                    }
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(&empty[sA]);
                        if (spt == 2) mbar_arrive(&empty[sB]);
                    }
                }
            }
        }
        // every warp's partials of this group are in: add them in warp order and store
        consumer_sync();
        const uint32_t per_tile = 16 * L.nc;
        auto total = [&](uint32_t tl, uint32_t r, uint32_t col) {
            const float *src = red + (size_t)tl * kGemvWarps * per_tile + r * L.nc + col;
            float sum = 0.f;
#pragma unroll
            for (int w = 0; w < kGemvWarps; w++) sum += src[(size_t)w * per_tile];
            return sum;
        };
        if (G.nranks == 0) {
            // sixteen threads take the rows of one (tile, column)
            for (uint32_t i = tid >> 4; i < gn * (SEP ? 1u : L.nc); i += kConsumers / 16) {
                const uint32_t tl = SEP ? i : i * L.nc_inv >> 16, col = SEP ? 0u : i - tl * L.nc;
                const float sum = total(tl, tid & 15, col);
                if constexpr (CL) {
                    part[((gb + tl) * L.nc + col) * 16 + (tid & 15)] = sum;  // this CTA's share of K
                    continue;
                }
                const GemvSeg sg = gemv_segment(p, t0 + gb + tl);
                const uint32_t row = (t0 + gb + tl - sg.tile0) * 16 + (tid & 15);
                if (row < sg.m) sg.out[(size_t)col * sg.m + row] = sum;
            }
        } else {
            // Row shards: an item is four consecutive rows of one column for one rank, stored
            // as one 16-byte word into that rank's copy of the whole output; the ranks of a
            // run of rows are taken by different threads so that their stores go out side by side.
            const uint32_t runs = gn * 4 * L.nc;  // (tile, four-row run, column)
            for (uint32_t i = tid; i < runs * G.nranks; i += kConsumers) {
                const uint32_t rk = i / runs, j = i % runs;
                const uint32_t tl = j / (4 * L.nc), r0 = (j / L.nc) % 4 * 4, col = j % L.nc;
                float sum[4];
#pragma unroll
                for (int e = 0; e < 4; e++) sum[e] = total(tl, r0 + e, col);
                const GemvSeg sg = gemv_segment(p, t0 + gb + tl);
                const uint32_t row = (t0 + gb + tl - sg.tile0) * 16 + r0;
                if (row >= sg.m) continue;
                float *dst = G.out[sg.index][rk] + (size_t)col * G.m_total[sg.index] + G.row_first[sg.index] + row;
                if (row + 4 <= sg.m && ((uintptr_t)dst & 15) == 0) {
                    *reinterpret_cast<float4 *>(dst) = make_float4(sum[0], sum[1], sum[2], sum[3]);
                } else {
                    for (uint32_t e = 0; e < 4 && row + e < sg.m; e++) dst[e] = sum[e];
                }
            }
        }
        if (gb + L.group < ntl) consumer_sync();  // before the buffer is zeroed again
    }
    if constexpr (CL) {
        // The cluster's CTAs have the same tiles: each adds up every so many-th (tile, column), in rank
        // order, reading the others' shares from their shared memory, and stores it.
        namespace cg = cooperative_groups;
        cg::cluster_group cl = cg::this_cluster();
        cl.sync();
        for (uint32_t j = ((tid >> 4) << clog) + rank; j < ntl * L.nc; j += kConsumers / 16 << clog) {
            float sum = 0.f;
            for (uint32_t q = 0; q < 1u << clog; q++) sum += cl.map_shared_rank(part, q)[j * 16 + (tid & 15)];
            const uint32_t tl = j / L.nc, col = j - tl * L.nc;
            const GemvSeg sg = gemv_segment(p, t0 + tl);
            const uint32_t row = (t0 + tl - sg.tile0) * 16 + (tid & 15);
            if (row < sg.m) sg.out[(size_t)col * sg.m + row] = sum;
        }
        cl.sync();  // nobody leaves while its shares may still be read
    }
    // Row shards: nobody fences or waits here.  The count the local counter has to reach for
    // the exchanges launched so far goes up by one per rank; whoever waits next reads it after
    // this kernel is complete.
    if (G.nranks && blockIdx.x == 0 && tid == 0) G.epoch[0] += G.nranks;
}

template <int TY, int MODE, int XDT, bool CL>
static cudaError_t launch_c(const GemvArgs &a, const GemvLayout &L, const GemvGather &G, uint32_t ctas, cudaStream_t s, int dev) {
    static bool attr_set[64] = {};  // the opt-in is per device
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (!attr_set[dev]) {
        cudaError_t e = cudaFuncSetAttribute(gemv_kernel<TY, MODE, XDT, CL>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSharedBudget);
        if (e != cudaSuccess) return e;
        attr_set[dev] = true;
    }
    return launch_pdl(gemv_kernel<TY, MODE, XDT, CL>, ctas, G.nranks ? kGemvThreadsMax : kGemvThreads, L.smem_bytes, s, 1u << L.clog, a, L, G);
}
template <int TY, int MODE, int XDT>
static cudaError_t launch_d(const GemvArgs &a, const GemvLayout &L, const GemvGather &G, uint32_t ctas, cudaStream_t s, int dev) {
    if constexpr (MODE == M_SEP)
        if (L.clog) return launch_c<TY, MODE, XDT, true>(a, L, G, ctas, s, dev);
    return launch_c<TY, MODE, XDT, false>(a, L, G, ctas, s, dev);
}
template <int TY, int MODE>
static cudaError_t launch_t(GemvArgs a, const GemvGather &G, int xdt, cudaStream_t s, int sms, int dev) {
    GemvLayout L;
    uint32_t ctas;
    if (!gemv_plan(TY, a.row_bytes, a.nunit, a.n, MODE, a.tiles, sms, G.nranks != 0, a, L, ctas)) return cudaErrorInvalidConfiguration;
    switch (xdt) {
    case DT_F16: return launch_d<TY, MODE, DT_F16>(a, L, G, ctas, s, dev);
    case DT_BF16: return launch_d<TY, MODE, DT_BF16>(a, L, G, ctas, s, dev);
    default: return launch_d<TY, MODE, DT_F32>(a, L, G, ctas, s, dev);
    }
}

// rows that end inside a unit: never a row shard, and the element type goes with the mode
template <int TY>
static cudaError_t launch_r(GemvArgs a, int mode, int xdt, cudaStream_t s, int sms, int dev) {
    GemvLayout L;
    uint32_t ctas;
    const GemvGather none = {};
    if (!gemv_plan(TY, a.row_bytes, a.nunit, a.n, mode, a.tiles, sms, false, a, L, ctas)) return cudaErrorInvalidConfiguration;
    switch (xdt) {
    case DT_F16: return launch_d<TY, M_R3, DT_F16>(a, L, none, ctas, s, dev);
    case DT_BF16: return launch_d<TY, M_R3, DT_BF16>(a, L, none, ctas, s, dev);
    default: return launch_d<TY, M_R4, DT_F32>(a, L, none, ctas, s, dev);
    }
}

template <int TY>
static cudaError_t launch_ty(const GemvArgs &a, const GemvGather &G, int mode, int xdt, cudaStream_t s, int sms, int dev) {
    switch (mode) {
    case M_SEP: return launch_t<TY, M_SEP>(a, G, xdt, s, sms, dev);
    case M_W1: return launch_t<TY, M_W1>(a, G, xdt, s, sms, dev);
    case M_W2: return launch_t<TY, M_W2>(a, G, xdt, s, sms, dev);
    }
    if constexpr (TY == T_Q8_0 || TY == T_Q4_0 || TY == T_IQ4_NL || TY == T_Q2_0) {
        if (mode == M_R4 || mode == M_R3) return launch_r<TY>(a, mode, xdt, s, sms, dev);
    }
    return cudaErrorInvalidValue;
}

static bool group_fits(int ty, uint32_t k, uint32_t nseg, const uint32_t *m, const uint8_t *const *w,
                       const void *x, int xdt, uint32_t n, int sms) {
    if (nseg == 0 || nseg > (uint32_t)kGemvSegs || n == 0 || n > 8) return false;
    if ((uintptr_t)x % 16 || (k * (xdt == DT_F32 ? 4 : 2)) % 16) return false;
    uint32_t tiles = 0;
    for (uint32_t i = 0; i < nseg; i++) {
        if (m[i] == 0 || (uintptr_t)w[i] % 16) return false;
        tiles += (m[i] + 15) / 16;
    }
    GemvArgs a = {};
    GemvLayout L;
    const uint32_t row_bytes = k / block_elems(ty) * block_bytes(ty);
    for (uint32_t left = n, take; left; left -= take) {
        const int mode = gemv_mode(k, xdt, left, take);
        uint32_t ctas;
        if (!gemv_plan(ty, row_bytes, (k + 255) / 256, take, mode, tiles, sms, false, a, L, ctas)) return false;
    }
    return true;
}

bool gemv_group_supported(int ty, uint32_t k, uint32_t nseg, const uint32_t *m, const uint8_t *const *w,
                          const void *x, int xdt, uint32_t n, int sms) {
    return has_fast_kernels(ty) && k % 256 == 0 && group_fits(ty, k, nseg, m, w, x, xdt, n, sms);
}

bool gemv_fast_supported(int ty, uint32_t k, uint32_t m, const void *w, const void *x, int xdt, uint32_t n,
                         int sms) {
    const uint8_t *wp = (const uint8_t *)w;
    return gemv_group_supported(ty, k, 1, &m, &wp, x, xdt, n, sms);
}

bool gemv_ragged_supported(int ty, uint32_t k, uint32_t m, const void *w, const void *x, int xdt, uint32_t n, int sms) {
    if (ty != T_Q8_0 && ty != T_Q4_0 && ty != T_IQ4_NL && ty != T_Q2_0) return false;
    const uint8_t *wp = (const uint8_t *)w;
    return k % 256 != 0 && group_fits(ty, k, 1, &m, &wp, x, xdt, n, sms);
}

// One launch covers up to eight columns (four where rows are no multiple of 256 weights; more are
// run as passes over consecutive columns).  `nseg` matrices of the same type and K share every launch.
cudaError_t launch_gemv_group(int ty, uint32_t nseg, const uint8_t *const *w, const uint32_t *m, float *const *out,
                              uint32_t k, const void *x, int xdt, uint32_t n, int *status, cudaStream_t s,
                              int sms, int dev, uint64_t *launches, const GemvGatherPlan *gather) {
    if (nseg == 0 || nseg > (uint32_t)kGemvSegs) return cudaErrorInvalidValue;
    GemvArgs a = {};
    a.status = status; a.k = k;
    a.nunit = (k + 255) / 256;
    a.row_bytes = k / block_elems(ty) * block_bytes(ty);
    uint32_t tiles = 0;
    for (uint32_t i = 0; i < (uint32_t)kGemvSegs; i++) {
        const uint32_t j = i < nseg ? i : nseg - 1;  // unused slots repeat the last one
        a.w[i] = w[j];
        a.m[i] = m[j];
        if (i < nseg) tiles += (m[i] + 15) / 16;
        a.tile_end[i] = tiles;
    }
    a.tiles = tiles;
    GemvGather G = {};
    if (gather) {
        G.nranks = gather->nranks;
        G.epoch = gather->epoch;
        G.wait_arrivals = gather->wait_arrivals;
        G.sig_nranks = gather->sig_nranks;
        for (uint32_t r = 0; r < gather->sig_nranks; r++) G.sig_arrivals[r] = gather->sig_arrivals[r];
        G.wait_epoch = gather->wait_epoch;
    }
    const size_t xsz = xdt == DT_F32 ? 4 : 2;
    for (uint32_t c0 = 0; c0 < n;) {
        uint32_t take;
        const int mode = gemv_mode(k, xdt, n - c0, take);
        a.x = (const uint8_t *)x + (size_t)c0 * k * xsz;
        for (uint32_t i = 0; i < (uint32_t)kGemvSegs; i++) {
            const uint32_t j = i < nseg ? i : nseg - 1;
            a.out[i] = (out && out[j]) ? out[j] + (size_t)c0 * m[j] : nullptr;
            if (gather) {
                G.m_total[i] = gather->seg[j].m_total;
                G.row_first[i] = gather->seg[j].row_first;
                for (uint32_t r = 0; r < gather->nranks; r++)
                    G.out[i][r] = gather->seg[j].out[r] + (size_t)c0 * gather->seg[j].m_total;
            }
        }
        a.n = take;
        cudaError_t e;
        int count = gather ? 0 : launch_gemv_stream(ty, mode, a, xdt, s, sms, dev, ring_estimate(ty, mode, a, sms), e);
        if (!count) switch (count = 1, ty) {
        case T_Q4_K: e = launch_ty<T_Q4_K>(a, G, mode, xdt, s, sms, dev); break;
        case T_Q8_0: e = launch_ty<T_Q8_0>(a, G, mode, xdt, s, sms, dev); break;
        case T_Q4_0: e = launch_ty<T_Q4_0>(a, G, mode, xdt, s, sms, dev); break;
        case T_Q6_K: e = launch_ty<T_Q6_K>(a, G, mode, xdt, s, sms, dev); break;
        case T_Q5_K: e = launch_ty<T_Q5_K>(a, G, mode, xdt, s, sms, dev); break;
        case T_IQ4_NL: e = launch_ty<T_IQ4_NL>(a, G, mode, xdt, s, sms, dev); break;
        case T_Q2_0: e = launch_ty<T_Q2_0>(a, G, mode, xdt, s, sms, dev); break;
        case T_IQ2_XXS: e = launch_ty<T_IQ2_XXS>(a, G, mode, xdt, s, sms, dev); break;
        default: e = cudaErrorInvalidValue;
        }
        if (e != cudaSuccess) return e;
        if (launches) *launches += (uint64_t)count;
        if (gather) {  // a further pass over columns announces this pass's exchange and waits for it
            G.wait_arrivals = gather->arrivals[gather->rank];
            G.wait_epoch = gather->epoch;
            G.sig_nranks = gather->nranks;
            for (uint32_t r = 0; r < gather->nranks; r++) G.sig_arrivals[r] = gather->arrivals[r];
        }
        c0 += take;
    }
    return cudaSuccess;
}

__global__ void gather_wait_kernel(GemvGather G, int *status) {
    pdl_wait();
    if (G.sig_nranks) gather_signal(G.sig_arrivals, G.sig_nranks);
    if (G.wait_arrivals) gather_wait(G.wait_arrivals, G.wait_epoch, status);
}

cudaError_t launch_gather_wait(const GemvGatherPlan &plan, int *status, cudaStream_t s) {
    GemvGather G = {};
    G.wait_arrivals = plan.wait_arrivals;
    G.wait_epoch = plan.wait_epoch;
    G.sig_nranks = plan.sig_nranks;
    for (uint32_t r = 0; r < plan.sig_nranks; r++) G.sig_arrivals[r] = plan.sig_arrivals[r];
    gather_wait_kernel<<<1, 1, 0, s>>>(G, status);
    return cudaGetLastError();
}

cudaError_t launch_gemv_fast(int ty, const uint8_t *w, uint32_t k, uint32_t m, const void *x, int xdt,
                             uint32_t n, float *out, int *status, cudaStream_t s, int sms, int dev,
                             uint64_t *launches) {
    return launch_gemv_group(ty, 1, &w, &m, &out, k, x, xdt, n, status, s, sms, dev, launches, nullptr);
}

}  // namespace okf
