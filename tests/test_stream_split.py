"""How a streaming matvec's units are dealt to warps, on the host: every unit of a CTA is in one warp's run, the parts of every tile that
a border cuts are added up once and in order, and the divisions by multiplication are exact over what a plan may hold; every plan the search finds
fits the shared memory that its kernel asks for."""
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
    for (uint32_t w = 0; w + 1 < NW; w++) {
        const uint32_t first = split.border<NW>(w), at = split.border<NW>(w + 1), tile = split.tile(at), lo = tile * units, hi = lo + units;
        if (!(at < split.all && at > lo && first <= lo)) continue;
        bad += !got[tile].empty();
        got[tile] = slot[2 * w + (first < lo)];
        for (uint32_t v = w + 1; v < NW && split.border<NW>(v) < hi; v++)
            if (split.border<NW>(v + 1) > split.border<NW>(v)) got[tile].insert(got[tile].end(), slot[2 * v].begin(), slot[2 * v].end());
    }
    for (uint32_t t = 0; t < tiles; t++) {
        bad += got[t].size() != units;
        for (uint32_t i = 0; i < got[t].size(); i++) bad += got[t][i] != t * units + i;
    }
    return bad;
}
template <int TY, int MODE> static unsigned plans(std::mt19937 &rng, unsigned &found) {
    unsigned bad = 0;
    const StreamRoom room = {{148, 74, 33, 15}, {296, 148, 71, 33}}, none = {{148, 0, 0, 0}, {296, 0, 0, 0}};
    for (int i = 0; i < 4000; i++) {
        const uint32_t nunit = 1 + rng() % (i % 4 ? 72 : 600), tiles = 1 + rng() % (i % 3 ? 1200 : 20000);
        const uint32_t n = MODE == M_SEP ? 1 : MODE == M_W2 ? 5 + rng() % 4 : 1 + rng() % 4;
        const StreamPlan p = stream_search<TY, MODE>(nunit, n, tiles, i & 1 ? room : none);
        if (!p.ok) continue;
        found++;
        const StreamLayout &L = p.L;
        const uint32_t size = 1u << L.clog, clusters = p.ctas / size, units = (nunit + size - 1) / size, per = (tiles + clusters - 1) / clusters;
        const uint32_t panel = (MODE == M_SEP ? 2 : n * mode_bytes(MODE)) * L.es, records = MODE == M_SEP ? 256 : units * n * wide_info_words(TY, mode_bytes(MODE)) * 4;
        bad += p.smem > (p.warps == 8 && p.ctas <= 148 ? kStreamAlone : stream_budget(p.warps)) || p.ctas % size || nunit < size || L.depth < 2 || L.depth > 4;
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
int main() {
    unsigned bad = 0, found = 0;
    for (uint32_t tiles = 1; tiles <= 40; tiles++)
        for (uint32_t units = 1; units <= 40; units++) bad += wrong<8>(tiles, units) + wrong<16>(tiles, units);
    std::mt19937 rng(3);
    bad += plans<T_Q4_K, M_SEP>(rng, found) + plans<T_Q4_K, M_W1>(rng, found) + plans<T_Q4_K, M_W2>(rng, found);
    bad += plans<T_Q6_K, M_SEP>(rng, found) + plans<T_Q8_0, M_W2>(rng, found) + plans<T_Q8_0, M_R4>(rng, found) + plans<T_Q2_0, M_R3>(rng, found);
    bad += plans<T_IQ2_XXS, M_SEP>(rng, found) + plans<T_IQ2_XXS, M_W1>(rng, found) + plans<T_IQ2_XXS, M_W2>(rng, found);
    printf("%u %u\n", bad, found);
}
"""


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    d = tmp_path_factory.mktemp("split")
    (d / "model.cu").write_text(MODEL)
    subprocess.run([build.nvcc(), "-O2", "-std=c++17", "--expt-relaxed-constexpr", *build.ARCH, "-I", str(build.CSRC), str(d / "model.cu"), "-o", str(d / "model")],
                   check=True)
    return d / "model"


def test_units_and_plans(model):
    bad, found = map(int, subprocess.run([str(model)], check=True, capture_output=True, text=True).stdout.split())
    assert bad == 0 and found > 20000


def test_results_of_other_kernels_are_not_read_through_the_read_only_path():
    """The kernel may be resident while the one before it writes x (see test_launch_rules)."""
    text = (build.CSRC / "okf_gemv_stream.cu").read_text()
    assert "pdl_wait();" in text and "__ldg(" not in text and "__restrict__" not in text
    body = text[text.index("pdl_wait();"):]
    assert "dep_ptr(" in body[:200] and "stage_x_wide" in body and "stage_x_bytes" not in text[:text.index("pdl_wait();")]
