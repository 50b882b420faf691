"""Plans of prefill matmuls with clusters, on the host: chains of sums no longer than without, room left where the last clusters would start late, and for
every type that shares items every size of cluster and number of accumulators among the shapes of the GPU test; the plans a thread keeps."""
import subprocess

from chatokf_b200 import build
from test_gpu_tile_clusters import TYPES, shapes

MODEL = r"""
#include <cstdio>
#include <random>
#include "okf_gemm_plan.h"
using namespace okf;
int main() {
    std::mt19937 rng(5);
    const int types[] = {T_Q8_0, T_Q4_K, T_IQ2_XXS, T_Q2_0, T_Q4_0, T_Q5_K, T_Q6_K, T_IQ4_NL};
    const uint32_t room[9] = {0, 0, 74, 45, 33, 26, 22, 15, 15};
    unsigned bad = 0;
    for (int i = 0; i < 20000; i++) {
        const int ty = types[rng() % 8], xdt = (int)(rng() % 3);
        const uint32_t k = 64 * (1 + rng() % 272), m = 1 + rng() % (i % 2 ? 20000 : 4000), n = 1 + rng() % 1000;
        const size_t mem = i % 5 ? (size_t)64 << 20 : 0;
        const GemmPlan p = gemm_tc_search(ty, k, m, n, xdt, 148, mem, room), r = gemm_tc_search(ty, k, m, n, xdt, 148, mem);
        if (!p.cluster) continue;
        const uint32_t items = (m + 127) / 128 * ((n + p.tok - 1) / p.tok), units = (k + 255) / 256;
        bad += ty == T_Q4_0;
        // no longer chains of sums than without clusters (sums in tensor memory are cut off where fp32 would round)
        const double chain = r.dealt && !r.waves ? (double)r.dealt * units / r.dealers : units;
        bad += (units + p.cluster - 1) / p.cluster > p.chains * (chain < 1 ? 1 : chain);
        // clusters of three and five leave room: the last ones of a full wave start late
        bad += (p.cluster == 3 || p.cluster == 5) && items * 16 > room[p.cluster] * 15;
        bad += !r.dealt && ((units < 8 && (p.cluster == 2 || items * 7 > room[p.cluster] * 6)) || (p.cluster == 2 && items == room[2]));
    }
    // what a thread kept, with clusters and without in turn, is what a search finds
    for (int i = 0; i < 6000; i++) {
        const int ty = types[i % 3], xdt = DT_F16;
        const uint32_t k = 256 * (4 + i % 31), m = 500 + 300 * (i % 7), n = 20 + 30 * (i % 5), *r = i & 1 ? room : nullptr;
        const GemmPlan p = gemm_tc_plan(ty, k, m, n, xdt, 148, (size_t)64 << 20, r), q = gemm_tc_search(ty, k, m, n, xdt, 148, (size_t)64 << 20, r);
        bad += p.tok != q.tok || p.cluster != q.cluster || p.chains != q.chains || p.dealt != q.dealt || p.dealers != q.dealers || p.floats != q.floats;
    }
    printf("%u\n", bad);
    int ty;
    uint32_t k, m, n;
    while (scanf("%d %u %u %u", &ty, &k, &m, &n) == 4) {
        const GemmPlan p = gemm_tc_search(ty, k, m, n, DT_F16, 148, (size_t)64 << 20, room);
        printf("%u %u\n", p.cluster, p.chains);
    }
}
"""


def test_clusters(tmp_path):
    (tmp_path / "model.cu").write_text(MODEL)
    subprocess.run([build.nvcc(), "-O2", "-std=c++17", *build.ARCH, "-I", str(build.CSRC), str(tmp_path / "model.cu"), "-o", str(tmp_path / "model")], check=True)
    asked = [(ty, k, m, n) for ty in TYPES for k, m, n in shapes(ty)]
    out = subprocess.run([str(tmp_path / "model")], input="".join(f"{int(t)} {k} {m} {n}\n" for t, k, m, n in asked), check=True, capture_output=True,
                         text=True).stdout.split("\n")
    assert out[0] == "0"
    plans = dict(zip(asked, (tuple(map(int, line.split())) for line in out[1:])))
    for ty in TYPES:
        mine = [plans[a] for a in asked if a[0] == ty]
        assert {c for c, _ in mine} == {2, 3, 4, 5, 6, 7, 8} and {a for _, a in mine} == {1, 2, 4}, (ty, mine)
