// Decode matvec whose warps stream weights for themselves (1..8 activation columns, every block type).
//
// The arithmetic is that of okf_gemv.cu (okf_gemv_unit.cuh, okf_gemv_wide.cuh); what differs is who takes which unit and how it gets
// there.  There all eight warps of a CTA share every stage that a producer fills: per stage and warp some 80 to 300 instructions
// of bookkeeping (which segment, how many units, barriers, sums into shared memory and out again) stand against one or two units of 120 to 300.
// And where rows do not come in whole, a bulk copy per row segment takes its warp 48 ns whatever its size, so K cannot be cut
// fine.  Here
//   - a CTA's units, tile after tile, are cut into eight equal runs, one a warp (sixteen for up to eight columns of large matrices).
//     A warp keeps its sums in registers through a tile; a tile that lies in its run whole is stored from there, the parts of a
//     tile that a border cuts (one or two a warp) meet in shared memory when all is done;
//   - a warp copies its own units with cp.async into a ring of its own, two to four stages of 16 row segments, and waits for its own
//     copies: no barriers, no producer.  144-byte segments come at 4.6 TB/s this way; by bulk copies, a row each, at 0.45 (0.9 with two
//     CTAs an SM), by a tensor-map box of 16 rows at 1.1 (2.0);
//   - K may be cut into slices of a few units: clusters of 2 to 8 CTAs share tiles, each with its slice of x, which it alone stages.
// What bounds it: instruction issue for several columns and the looked-up types (60 % of the slots, ALU pipe 45 to 62 %), x's staging
// (some 110 instructions per column and unit), at one column of large matrices the copies themselves (4.9 TB/s; okf_gemv.cu's bulk copies
// of whole rows reach 6.1 and keep those, see ring_us).
// us in chains of launches, there and here: Q4_K 2560 -> 2 x 9728 at 1 / 4 / 8 columns 9.0 / 11.5 / 17.3 and 8.3 / 9.4 / 12.3,
// 9728 -> 2560 at 4 / 8 13.4 / 19.8 and 8.4 / 10.8; IQ2_XXS 17408 -> 5120 at 1 / 4 / 8 20.2 / 31 / 73 and 15.4 / 19.8 / 25; Q8_0 14336 ->
// 4096 at 4 34.8 and 19.2; Q4_0 1056 -> 5003 at 3 5.0 and 4.3.
// Tried: three CTAs to an SM (80 registers; Q4_K 2560 -> 2 x 9728, one column 9.4 against 8.6), two units of 144 bytes a stage (no change), sixteen
// warps for up to four columns (9.6 against 9.4; no room for the next launch's first copies).
#include <cooperative_groups.h>

#include <mutex>

#include "okf_gemv_stream.h"
#include "okf_kernels.h"

namespace okf {

__device__ __forceinline__ void cp_async16(uint32_t dst, const uint8_t *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <int TY, int MODE, int XDT, uint32_t NW>
__global__ void __launch_bounds__(NW * 32, 16 / NW) stream_kernel(const __grid_constant__ GemvArgs p, const __grid_constant__ StreamLayout L) {
    using S = StreamGeom<TY, MODE>;
    using W = WideMode<MODE>;
    constexpr bool SEP = MODE == M_SEP;
    constexpr uint32_t UB = S::ub;
    extern __shared__ __align__(128) uint8_t smem[];
    const uint32_t smem32 = smem_u32(smem);
    const uint32_t tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31, g = lane >> 2, c = lane & 3;
    const uint32_t clog = L.clog, rank = blockIdx.x & ((1u << clog) - 1), cid = blockIdx.x >> clog;
    const uint32_t t0 = L.tile_first + cid * L.tiles_each + min(cid, L.tiles_more), ntl = L.tiles_each + (cid < L.tiles_more ? 1u : 0u);
    const uint32_t ubeg = p.nunit * rank >> clog, nun = (p.nunit * (rank + 1) >> clog) - ubeg;
    // this warp's units of the CTA's tiles laid end to end
    const StreamSplit split(ntl, nun, nun == p.nunit >> clog ? L.unit_inv : L.unit_inv_more);
    const uint32_t first = split.border<NW>(warp), last = split.border<NW>(warp + 1);
    const uint32_t tile_first = split.tile(first), unit_first = first - tile_first * nun;

    pdl_launch_dependents();
    // ---- copies: lane (g, c) takes every fourth 16 bytes of rows g and g + 8
    const uint32_t ring = smem32 + warp * L.depth * S::stage + g * S::pitch;
    uint32_t ct = tile_first, cu = unit_first, cleft = last - first;  // what is copied next
    const uint8_t *r0 = nullptr, *r1 = nullptr;
    auto rows_of = [&](uint32_t t) {
        const GemvSeg sg = gemv_segment(p, t0 + t);
        const uint32_t row = (t0 + t - sg.tile0) * 16 + g;
        const uint8_t *w = sg.w + (size_t)ubeg * UB;
        r0 = w + (size_t)min(row, sg.m - 1) * p.row_bytes;
        r1 = w + (size_t)min(row + 8, sg.m - 1) * p.row_bytes;
    };
    auto copy = [&](uint32_t slot) {
        if (cleft) {
            const uint32_t len = S::cb == 1 ? 1u : min(min(S::cb, nun - cu), cleft);
            const uint32_t at = ring + slot * S::stage;
            uint32_t bytes = len * UB;
            if constexpr (S::rag) bytes = min(bytes, p.row_bytes - (ubeg + cu) * UB);  // the last unit of a row may not be whole
#pragma unroll
            for (uint32_t h = 0; h < 2; h++) {
                // from the 32-byte boundary below the segment, to where the segment itself starts 16 bytes into its row (and as
                // many as it lies behind a 16-byte boundary): its banks do not depend on where rows start
                const uintptr_t src = reinterpret_cast<uintptr_t>(h ? r1 : r0) + cu * UB;
                const uint8_t *from = reinterpret_cast<const uint8_t *>(src & ~(uintptr_t)31) + 16 * c;
                const uint32_t end = ((uint32_t)src & 31u) + bytes, to = at + h * 8 * S::pitch + 16 - ((uint32_t)src & 16u) + 16 * c;
#pragma unroll
                for (uint32_t i = 0; i < (S::bytes + 63) / 64; i++)
                    if ((S::cb == 1 && !S::rag && 64 * i + 64 <= UB) || 64 * i + 16 * c < end) cp_async16(to + 64 * i, from + 64 * i);
            }
            cu += len;
            cleft -= len;
            if (cu == nun && cleft) {
                cu = 0;
                rows_of(++ct);
            }
        }
        cp_async_commit();
    };
    if (cleft) rows_of(ct);
    uint32_t q0 = (uint32_t)reinterpret_cast<uintptr_t>(r0) & 15u, q1 = (uint32_t)reinterpret_cast<uintptr_t>(r1) & 15u;  // (of what is read next)
#pragma unroll 1
    for (uint32_t s = 0; s < L.depth; s++) copy(s);

    if constexpr (SEP)
        if (tid < 64) sts32(smem32 + L.slot_off - 256 + tid * 4, 0u);
    if constexpr (TY == T_IQ2_XXS) {
        // the look-up tables, every entry `tab_copies` times side by side (see Iq2Tab), 16 bytes a store
        const uint32_t per = L.tab_copies / 4, sh = 31 - __clz(per);
        for (uint32_t i = tid; i < 384u * per; i += NW * 32) {
            const uint32_t v = g_iq2_selectors.v[i >> sh];
            *reinterpret_cast<uint4 *>(smem + L.tab_off + i * 16) = make_uint4(v, v, v, v);
        }
    }
    Iq2Tab tab = {0, 0, 0};
    if constexpr (TY == T_IQ2_XXS) {
        tab.stride = L.tab_copies * 4;
        tab.code = smem32 + L.tab_off + (lane & (L.tab_copies - 1)) * 4;
        tab.sign = tab.code + 256 * tab.stride;
    }
    const SepConst KC = sep_const<TY>(c);
    const bool sep_active = (g >> 1) == c;
    const uint32_t xbase32 = sep_active ? smem32 + L.xs_off + (g & 1) * L.es + c * kSepQuarter
                                        : smem32 + L.slot_off - 256 + ((5 * (g >> 1) + 1) & 7) * 16;
    const uint32_t xstride32 = sep_active ? kSepUnit : 0u;
    const uint32_t rec32 = smem32 + L.xs_off + c * kSepQuarter + 64;
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
            ws32[i] = info32 + (fed < p.n ? fed : 0u) * kInfo + 4 + (g & 1) * kPlane + 4 * word;
            ws_lo = (2 - (g & 1)) * kPlane;
        }
    }

    pdl_wait();
    const void *x = dep_ptr(reinterpret_cast<const uint8_t *>(p.x));
    if constexpr (SEP) stage_x_bytes<TY, XDT, NW>(smem32 + L.xs_off, L.es, x, ubeg, nun, tid);
    else stage_x_wide<TY, MODE, XDT, NW>(smem32 + L.xs_off, L.es, info32, x, p.k, L.nc, ubeg, nun, tid);
    __syncthreads();

    constexpr int NV = SEP ? 1 : W::vals;
    float acc[NV][2], sum[NV][2];
#pragma unroll
    for (int i = 0; i < NV; i++) acc[i][0] = acc[i][1] = sum[i][0] = sum[i][1] = 0.f;
    uint32_t t = tile_first, u = unit_first, begun = unit_first, left = last - first, slot = 0;
    while (left) {
        if (L.depth == 2) cp_async_wait<1>();
        else if (L.depth == 3) cp_async_wait<2>();
        else cp_async_wait<3>();
        __syncwarp();
        const uint32_t len = S::cb == 1 ? 1u : min(min(S::cb, nun - u), left);
        uint32_t wa = ring + slot * S::stage + 16, wb = wa + 8 * S::pitch;
        if constexpr (!S::aligned) {
            wa += (q0 + u * UB) & 15u;
            wb += (q1 + u * UB) & 15u;
        }
#pragma unroll
        for (uint32_t i = 0; i < S::cb; i++) {
            if (i < len) {
                if constexpr (SEP) {
                    const uint32_t xa = xbase32 + u * xstride32, ia = rec32 + u * kSepUnit;
                    const uint4 v0 = lds128(xa), v1 = lds128(xa + 16), v2 = lds128(xa + 32), v3 = lds128(xa + 48);
                    const uint32_t xf[16] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w, v2.x, v2.y, v2.z, v2.w, v3.x, v3.y, v3.z, v3.w};
                    const uint4 xi = lds128(ia);
                    const uint4 xj = TY == T_Q6_K ? lds128(ia + L.es) : make_uint4(0u, 0u, 0u, 0u);
                    unit_sep<TY>(wa, wb, KC, tab, xf, xi, xj, acc[0]);
                } else {
                    const uint32_t xoff = u * kXqUnit, ioff = u * L.nc * kInfo;
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
                    unit_wide<TY, MODE>(wa, wb, c, X, tab, p.k / 32 - (ubeg + u) * 8, acc);
                    // Rows that end inside a unit have x as it is, so the rounding of these sums is all there is: a tile's units, which one warp may have all of, are
                    // added up in fours first (Q2_0 17280 -> 20000, one column, rms error 1.11e-7 in one run, 0.83e-7 in fours, 0.82e-7 in okf_gemv.cu's kernel; 0.96 to 0.98
                    // of that one's over 163 shapes of 48 and 500; no difference in time).
                    if constexpr (W::rag)
                        if ((u & 3) == 3) {
#pragma unroll
                            for (int r = 0; r < NV; r++) {
                                sum[r][0] += acc[r][0];
                                sum[r][1] += acc[r][1];
                                acc[r][0] = acc[r][1] = 0.f;
                            }
                        }
                }
                wa += UB;
                wb += UB;
                u++;
            }
        }
        left -= len;
        if (u == nun || left == 0) {
            // a tile that this warp has from end to end goes out from here, a part of one into one of the warp's two slots
            const bool whole = begun == 0 && u == nun;
            if constexpr (W::rag) {
#pragma unroll
                for (int i = 0; i < NV; i++) {
                    acc[i][0] += sum[i][0];
                    acc[i][1] += sum[i][1];
                    sum[i][0] = sum[i][1] = 0.f;
                }
            }
            if constexpr (SEP) {
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    acc[0][e] += __shfl_xor_sync(0xffffffffu, acc[0][e], 1);
                    acc[0][e] += __shfl_xor_sync(0xffffffffu, acc[0][e], 2);
                }
            }
            if (whole && clog == 0) {
                const GemvSeg sg = gemv_segment(p, t0 + t);
                const uint32_t row = (t0 + t - sg.tile0) * 16 + g;
                if constexpr (SEP) {
                    if (c < 2 && row + 8 * c < sg.m) sg.out[row + 8 * c] = c ? acc[0][1] : acc[0][0];
                } else {
#pragma unroll
                    for (int i = 0; i < NV; i++)
                        if (4 * i + c < L.nc) {
                            float *o = sg.out + (size_t)(4 * i + c) * sg.m + row;
                            if (row < sg.m) o[0] = acc[i][0];
                            if (row + 8 < sg.m) o[8] = acc[i][1];
                        }
                }
            } else {
                const uint32_t dst = smem32 + (whole ? L.part_off + t * L.nc * 64 : L.slot_off + (warp * 2 + (t != tile_first)) * L.nc * 64) + g * 4;
                if constexpr (SEP) {
                    if (c < 2) sts32(dst + 32 * c, __float_as_uint(c ? acc[0][1] : acc[0][0]));
                } else {
#pragma unroll
                    for (int i = 0; i < NV; i++)
                        if (4 * i + c < L.nc) {
                            sts32(dst + (4 * i + c) * 64, __float_as_uint(acc[i][0]));
                            sts32(dst + (4 * i + c) * 64 + 32, __float_as_uint(acc[i][1]));
                        }
                }
            }
#pragma unroll
            for (int i = 0; i < NV; i++) acc[i][0] = acc[i][1] = 0.f;
            u = begun = 0;
            t++;
            if constexpr (!S::aligned) {
                if (left) {
                    const GemvSeg sg = gemv_segment(p, t0 + t);
                    const uint32_t row = (t0 + t - sg.tile0) * 16 + g, w = (uint32_t)reinterpret_cast<uintptr_t>(sg.w) + ubeg * UB;
                    q0 = w + min(row, sg.m - 1) * p.row_bytes;
                    q1 = w + min(row + 8, sg.m - 1) * p.row_bytes;
                }
            }
        }
        __syncwarp();
        copy(slot);
        slot = slot + 1 == L.depth ? 0 : slot + 1;
    }
    __syncthreads();
    // Tiles that borders between warps cut: the warps in front of those borders have them added up, in warp order, each its share of the columns.  (Left to
    // the first of them, up to seven parts of eight columns one after the other: rows of two to six units, 5 to 8 columns, 160 shapes, took 1.22 times as long;
    // IQ4_NL 1024 -> 209, 8 columns, 4.8 and 3.6 us.)
    const uint32_t tile = split.tile(last), lo = tile * nun;
    if (warp + 1 < NW && last < split.all && last > lo && (!SEP || first <= lo)) {  // (a single column is the first one's)
        uint32_t w0 = warp, w1 = warp + 1;  // the first and the last warp with a part
        if constexpr (!SEP)
            while (split.border<NW>(w0) > lo) w0--;
        while (w1 + 1 < NW && split.border<NW>(w1 + 1) < lo + nun) w1++;
        const float *slots = reinterpret_cast<const float *>(smem + L.slot_off) + (lane & 15);
        const GemvSeg sg = gemv_segment(p, t0 + tile);
        const uint32_t row = (t0 + tile - sg.tile0) * 16 + (lane & 15), slot0 = w0 * 2 + (split.border<NW>(w0) < lo);
        for (uint32_t col = (lane >> 4) + 2 * (warp - w0); col < L.nc; col += 2 * (w1 - w0)) {
            float sum = slots[(slot0 * L.nc + col) * 16];
            for (uint32_t v = w0 + 1; v <= w1; v++)
                if (split.border<NW>(v + 1) > split.border<NW>(v)) sum += slots[(v * 2 * L.nc + col) * 16];
            if (clog) reinterpret_cast<float *>(smem + L.part_off)[(tile * L.nc + col) * 16 + (lane & 15)] = sum;
            else if (row < sg.m) sg.out[(size_t)col * sg.m + row] = sum;
        }
    }
    if (clog) {
        namespace cg = cooperative_groups;
        cg::cluster_group cl = cg::this_cluster();
        cl.sync();
        float *part = reinterpret_cast<float *>(smem + L.part_off);
        for (uint32_t j = ((tid >> 4) << clog) + rank; j < ntl * L.nc; j += NW * 2 << clog) {
            float sum = 0.f;
            for (uint32_t q = 0; q < 1u << clog; q++) sum += cl.map_shared_rank(part, q)[j * 16 + (tid & 15)];
            const uint32_t tl = SEP ? j : j * L.nc_inv >> 16, col = SEP ? 0u : j - tl * L.nc;
            const GemvSeg sg = gemv_segment(p, t0 + tl);
            const uint32_t row = (t0 + tl - sg.tile0) * 16 + (tid & 15);
            if (row < sg.m) sg.out[(size_t)col * sg.m + row] = sum;
        }
        cl.sync();
    }
}

// What fits on the device, looked up once.
static bool stream_room(int dev, int sms, StreamRoom &room) {
    struct Known {
        std::once_flag once;
        bool ok = false;
        StreamRoom room;
    };
    static Known known[64];
    if (dev < 0 || dev >= 64) return false;
    Known &k = known[dev];
    std::call_once(k.once, [&] {
        auto one = stream_kernel<T_Q4_K, M_W2, DT_F32, 16>;
        auto two = stream_kernel<T_Q4_K, M_W2, DT_F32, 8>;
        if (cudaFuncSetAttribute(one, cudaFuncAttributeMaxDynamicSharedMemorySize, stream_budget(16)) != cudaSuccess ||
            cudaFuncSetAttribute(two, cudaFuncAttributeMaxDynamicSharedMemorySize, stream_budget(8)) != cudaSuccess) {
            (void)cudaGetLastError();  // not for whoever asks next
            return;
        }
        k.room.one[0] = (uint32_t)sms;
        k.room.two[0] = 2 * (uint32_t)sms;
        for (uint32_t clog = 1; clog < 4; clog++) {
            for (int w = 0; w < 2; w++) {
                cudaLaunchAttribute at;
                at.id = cudaLaunchAttributeClusterDimension;
                at.val.clusterDim.x = 1u << clog;
                at.val.clusterDim.y = at.val.clusterDim.z = 1;
                cudaLaunchConfig_t cfg = {};
                cfg.gridDim = dim3(2 * (uint32_t)sms << clog);
                cfg.blockDim = dim3(w ? 256 : 512);
                cfg.dynamicSmemBytes = stream_budget(w ? 8 : 16);
                cfg.attrs = &at;
                cfg.numAttrs = 1;
                int n = 0;
                if (cudaOccupancyMaxActiveClusters(&n, w ? (const void *)two : (const void *)one, &cfg) != cudaSuccess) {
                    (void)cudaGetLastError();
                    n = 0;  // none of that size
                }
                (w ? k.room.two : k.room.one)[clog] = (uint32_t)n;
            }
        }
        k.ok = true;
    });
    if (k.ok) room = k.room;
    return k.ok;
}

template <int TY, int MODE, int XDT, uint32_t NW>
static cudaError_t stream_go(const GemvArgs &a, const StreamPlan &p, const StreamLayout &L, uint32_t ctas, cudaStream_t s, int dev) {
    static bool attr_set[64] = {};  // the opt-in is per device
    if (!attr_set[dev]) {
        cudaError_t e = cudaFuncSetAttribute(stream_kernel<TY, MODE, XDT, NW>, cudaFuncAttributeMaxDynamicSharedMemorySize, NW == 8 ? kStreamAlone : stream_budget(NW));
        if (e != cudaSuccess) return e;
        attr_set[dev] = true;
    }
    return launch_kernel(p.early, stream_kernel<TY, MODE, XDT, NW>, ctas, NW * 32, p.smem, s, 1u << L.clog, a, L);
}
template <int TY, int MODE, int XDT>
static cudaError_t stream_warps(const GemvArgs &a, const StreamPlan &p, const StreamLayout &L, uint32_t ctas, cudaStream_t s, int dev) {
    if constexpr (MODE == M_W2)
        if (p.warps == 16) return stream_go<TY, MODE, XDT, 16>(a, p, L, ctas, s, dev);
    return stream_go<TY, MODE, XDT, 8>(a, p, L, ctas, s, dev);
}
template <int TY, int MODE, int XDT>
static cudaError_t stream_all(const GemvArgs &a, const StreamPlan &p, cudaStream_t s, int dev) {
    if (p.tiles == a.tiles) return stream_warps<TY, MODE, XDT>(a, p, p.L, p.ctas, s, dev);
    StreamLayout L = p.L;
    for (uint32_t first = 0; first < a.tiles; first += p.tiles) {
        const uint32_t tiles = a.tiles - first < p.tiles ? a.tiles - first : p.tiles, all = p.ctas >> L.clog, clusters = tiles < all ? tiles : all;
        L.deal(first, tiles, clusters);
        const cudaError_t e = stream_warps<TY, MODE, XDT>(a, p, L, clusters << L.clog, s, dev);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}
template <int TY, int MODE>
static int stream_launch(const GemvArgs &a, int xdt, const StreamRoom &room, cudaStream_t s, int dev, float other_us, cudaError_t &e) {
    const StreamPlan &p = stream_plan<TY, MODE>(a.nunit, a.n, a.tiles, room, dev);
    if (!p.ok || p.us >= other_us) return 0;
    if constexpr (MODE == M_R4) e = stream_all<TY, MODE, DT_F32>(a, p, s, dev);
    else if constexpr (MODE == M_R3) e = xdt == DT_F16 ? stream_all<TY, MODE, DT_F16>(a, p, s, dev) : stream_all<TY, MODE, DT_BF16>(a, p, s, dev);
    else if (xdt == DT_F16) e = stream_all<TY, MODE, DT_F16>(a, p, s, dev);
    else if (xdt == DT_BF16) e = stream_all<TY, MODE, DT_BF16>(a, p, s, dev);
    else e = stream_all<TY, MODE, DT_F32>(a, p, s, dev);
    return p.tiles == a.tiles ? 1 : (int)((a.tiles + p.tiles - 1) / p.tiles);
}
template <int TY>
static int stream_ty(int mode, const GemvArgs &a, int xdt, const StreamRoom &room, cudaStream_t s, int dev, float other_us, cudaError_t &e) {
    switch (mode) {
    case M_SEP: return stream_launch<TY, M_SEP>(a, xdt, room, s, dev, other_us, e);
    case M_W1: return stream_launch<TY, M_W1>(a, xdt, room, s, dev, other_us, e);
    case M_W2: return stream_launch<TY, M_W2>(a, xdt, room, s, dev, other_us, e);
    }
    if constexpr (TY == T_Q8_0 || TY == T_Q4_0 || TY == T_IQ4_NL || TY == T_Q2_0) {
        if (mode == M_R4) return stream_launch<TY, M_R4>(a, xdt, room, s, dev, other_us, e);
        if (mode == M_R3) return stream_launch<TY, M_R3>(a, xdt, room, s, dev, other_us, e);
    }
    return 0;
}
int launch_gemv_stream(int ty, int mode, const GemvArgs &a, int xdt, cudaStream_t s, int sms, int dev, float other_us, cudaError_t &e) {
    StreamRoom room;
    if (!stream_room(dev, sms, room)) return 0;
    switch (ty) {
    case T_Q4_K: return stream_ty<T_Q4_K>(mode, a, xdt, room, s, dev, other_us, e);
    case T_Q8_0: return stream_ty<T_Q8_0>(mode, a, xdt, room, s, dev, other_us, e);
    case T_Q4_0: return stream_ty<T_Q4_0>(mode, a, xdt, room, s, dev, other_us, e);
    case T_Q6_K: return stream_ty<T_Q6_K>(mode, a, xdt, room, s, dev, other_us, e);
    case T_Q5_K: return stream_ty<T_Q5_K>(mode, a, xdt, room, s, dev, other_us, e);
    case T_IQ4_NL: return stream_ty<T_IQ4_NL>(mode, a, xdt, room, s, dev, other_us, e);
    case T_Q2_0: return stream_ty<T_Q2_0>(mode, a, xdt, room, s, dev, other_us, e);
    case T_IQ2_XXS: return stream_ty<T_IQ2_XXS>(mode, a, xdt, room, s, dev, other_us, e);
    default: return 0;
    }
}
}  // namespace okf
