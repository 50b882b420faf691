"""How a streaming matvec is cut, on the host: into launches where the sums of all tiles do not fit, and into runs of units a warp, whose cut tiles
are added up in order, every column once; every plan fits the shared memory that its kernel asks for, and no whole row goes without one."""
import subprocess

import pytest

from chatokf_b200 import build

MODEL = r"""
#include <cstdio>
#include <random>
#include <vector>
#include "okf_gemv_stream.h"
using namespace okf;

// What the kernel does behind its loop, with counts in the place of sums: units added up per tile.
template <uint32_t NW> static unsigned wrong(uint32_t tiles, uint32_t units) {
    const StreamSplit split(tiles, units, stream_inv(units));
    std::vector<std::vector<uint32_t>> got(tiles);  // units in the order they are added
    std::vector<std::vector<uint32_t>> slot(2 * NW);
    unsigned bad = 0;
    for (uint32_t w = 0; w < NW; w++) {
        const uint32_t first = split.border<NW>(w), last = split.border<NW>(w + 1);
        bad += first > last || split.tile(first) != first / units;
        for (uint32_t v = first; v < last;) {
            const uint32_t t = v / units, end = std::min(last, (t + 1) * units);
            std::vector<uint32_t> part;
            for (; v < end; v++) part.push_back(v);
            if (part.size() == units) got[t] = part;  // whole: stored from the warp
            else slot[2 * w + (t != first / units)] = part;
        }
    }
    bad += split.border<NW>(0) != 0 || split.border<NW>(NW) != tiles * units;
    for (uint32_t nc : {1u, 3u, 8u}) {
        std::vector<unsigned> taken(tiles * nc);  // how many warps add a column of a tile up
        for (uint32_t w = 0; w + 1 < NW; w++) {
            const uint32_t last = split.border<NW>(w + 1), tile = split.tile(last), lo = tile * units, hi = lo + units;
            if (!(last < split.all && last > lo)) continue;
            uint32_t w0 = w, w1 = w + 1;
            while (split.border<NW>(w0) > lo) w0--;
            while (w1 + 1 < NW && split.border<NW>(w1 + 1) < hi) w1++;
            std::vector<uint32_t> sum = slot[2 * w0 + (split.border<NW>(w0) < lo)];
            for (uint32_t v = w0 + 1; v <= w1; v++)
                if (split.border<NW>(v + 1) > split.border<NW>(v)) sum.insert(sum.end(), slot[2 * v].begin(), slot[2 * v].end());
            for (uint32_t half = 0; half < 2; half++)
                for (uint32_t col = half + 2 * (w - w0); col < nc; col += 2 * (w1 - w0)) taken[tile * nc + col]++;
            bad += !got[tile].empty() && got[tile] != sum;
            got[tile] = sum;
        }
        for (uint32_t t = 0; t < tiles; t++) {
            bool cut = false;
            for (uint32_t w = 1; w < NW; w++) cut |= split.border<NW>(w) > t * units && split.border<NW>(w) < (t + 1) * units;
            for (uint32_t c = 0; c < nc; c++) bad += taken[t * nc + c] != cut;
        }
    }
    for (uint32_t t = 0; t < tiles; t++) {
        bad += got[t].size() != units;
        for (uint32_t i = 0; i < got[t].size(); i++) bad += got[t][i] != t * units + i;
    }
    return bad;
}
static unsigned late = 0;
template <int TY, int MODE> static unsigned plans(std::mt19937 &rng, unsigned &found) {
    unsigned bad = 0;
    const StreamRoom room = {{148, 74, 33, 15}, {296, 148, 71, 33}}, none = {{148, 0, 0, 0}, {296, 0, 0, 0}};
    for (int i = 0; i < 4000; i++) {
        const uint32_t nunit = 1 + rng() % (i % 4 ? 72 : 600), wanted = 1 + rng() % (i % 3 ? 1200 : 20000);
        const uint32_t n = MODE == M_SEP ? 1 : MODE == M_W2 ? 5 + rng() % 4 : 1 + rng() % 4;
        const StreamRoom &fits = i & 1 ? room : none;
        const StreamPlan p = stream_launches<TY, MODE>(nunit, n, wanted, fits);
        if (!p.ok) continue;
        const uint32_t tiles = p.tiles;  // of a launch
        bad += tiles == 0 || tiles > wanted;
        found++;
        StreamLayout rest = p.L;  // the last launch takes what is left of the matrix, in as many clusters at most
        const uint32_t left = wanted % tiles ? wanted % tiles : tiles, fit = left < p.ctas >> p.L.clog ? left : p.ctas >> p.L.clog;
        rest.deal(wanted - left, left, fit);
        bad += rest.tile_first + rest.tiles_each * fit + rest.tiles_more != wanted || rest.tiles_each > p.L.tiles_each || rest.tiles_each + !!rest.tiles_more > p.L.tiles_each + !!p.L.tiles_more;
        // grids that take every SM in clusters of four and eight, and last, wait for their predecessors; nothing else does
        bad += p.early != !(p.ctas >> p.L.clog > fits.one[p.L.clog] && p.L.clog >= 2 && p.us >= kStreamLate);
        late += !p.early;
        const StreamLayout &L = p.L;
        const uint32_t size = 1u << L.clog, clusters = p.ctas / size, units = (nunit + size - 1) / size, per = (tiles + clusters - 1) / clusters;
        const uint32_t panel = (MODE == M_SEP ? 2 : n * mode_bytes(MODE)) * L.es, records = MODE == M_SEP ? 256 : units * n * wide_info_words(TY, mode_bytes(MODE)) * 4;
        // only where there is an SM for every CTA of a cluster does a grid ask for SMs of its own: the last clusters would wait for the first else
        bad += p.smem > (p.warps == 8 && clusters <= fits.one[L.clog] ? kStreamAlone : stream_budget(p.warps)) || p.ctas % size || nunit < size || L.depth < 2 || L.depth > 4;
        bad += L.tiles_each * clusters + L.tiles_more != tiles || L.tiles_more >= clusters || L.tiles_each == 0;
        bad += p.warps * L.depth * StreamGeom<TY, MODE>::stage > L.xs_off || L.xs_off % 128 || L.xs_off + panel > L.info_off || L.slot_off % 128;
        bad += L.info_off + records > L.slot_off || L.slot_off + p.warps * 2 * n * 64 > L.part_off || L.part_off + (size > 1 ? per * n * 64 : 0) > L.tab_off;
        bad += L.tab_off + 1536 * L.tab_copies > p.smem || (TY == T_IQ2_XXS) != (L.tab_copies >= 16);
        bad += !stream_exact(per, units, n);
        for (uint32_t j = 0; j < 20; j++) {
            const uint32_t few = nunit / size, v = rng() % (per * units + 1), c = rng() % (per * n);
            bad += StreamSplit(per, few, L.unit_inv).tile(v) != v / few || StreamSplit(per, few + 1, L.unit_inv_more).tile(v) != v / (few + 1);
            bad += (c * L.nc_inv >> 16) != c / n;
        }
    }
    return bad;
}
// whole rows of up to 112 units at two to eight columns: there is a plan, and it has all of x in shared memory
template <int TY> static unsigned declined() {
    const StreamRoom room = {{148, 74, 33, 15}, {296, 148, 71, 33}};
    unsigned no = 0;
    for (uint32_t nunit = 1; nunit <= 112; nunit++)
        for (uint32_t tiles = 16; tiles <= 16384; tiles += tiles / 8)
            for (uint32_t n = 2; n <= 8; n++) no += !(n <= 4 ? stream_launches<TY, M_W1>(nunit, n, tiles, room) : stream_launches<TY, M_W2>(nunit, n, tiles, room)).ok;
    return no;
}
int main() {
    unsigned bad = 0, found = 0;
    bad += declined<T_Q8_0>() + declined<T_Q4_K>() + declined<T_IQ2_XXS>() + declined<T_Q2_0>() + declined<T_Q4_0>() + declined<T_Q5_K>() + declined<T_Q6_K>() + declined<T_IQ4_NL>();
    for (uint32_t tiles = 1; tiles <= 40; tiles++)
        for (uint32_t units = 1; units <= 40; units++) bad += wrong<8>(tiles, units) + wrong<16>(tiles, units);
    std::mt19937 rng(3);
    bad += plans<T_Q4_K, M_SEP>(rng, found) + plans<T_Q4_K, M_W1>(rng, found) + plans<T_Q4_K, M_W2>(rng, found);
    bad += plans<T_Q6_K, M_SEP>(rng, found) + plans<T_Q8_0, M_W2>(rng, found) + plans<T_Q8_0, M_R4>(rng, found) + plans<T_Q2_0, M_R3>(rng, found);
    bad += plans<T_IQ2_XXS, M_SEP>(rng, found) + plans<T_IQ2_XXS, M_W1>(rng, found) + plans<T_IQ2_XXS, M_W2>(rng, found);
    printf("%u %u %u\n", bad, found, late);
}
"""


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    d = tmp_path_factory.mktemp("launches")
    (d / "model.cu").write_text(MODEL)
    subprocess.run([build.nvcc(), "-O2", "-std=c++17", "--expt-relaxed-constexpr", *build.ARCH, "-I", str(build.CSRC), str(d / "model.cu"), "-o", str(d / "model")],
                   check=True)
    return d / "model"


def test_launches(model):
    bad, found, late = map(int, subprocess.run([str(model)], check=True, capture_output=True, text=True).stdout.split())
    assert bad == 0 and found > 20000 and late > 100
