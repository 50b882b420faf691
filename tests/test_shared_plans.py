"""Plans of prefill matmuls with clusters, on the host: no partial tiles, no more clusters than there is room for, units for every CTA, k-blocks for every accumulator, and a
search without room for any finds what it found before there were clusters."""
import subprocess

from chatokf_b200 import build

MODEL = r"""
#include <cstdio>
#include <random>
#include "okf_gemm_plan.h"
using namespace okf;
int main() {
    std::mt19937 rng(5);
    const int types[] = {T_Q8_0, T_Q4_K, T_IQ2_XXS, T_Q2_0, T_Q4_0, T_Q5_K, T_Q6_K, T_IQ4_NL};
    const uint32_t room[9] = {0, 0, 74, 45, 33, 26, 22, 15, 15}, none[9] = {};
    unsigned bad = 0, sizes = 0, accs = 0;
    for (int i = 0; i < 20000; i++) {
        const int ty = types[rng() % 8], xdt = (int)(rng() % 3);
        const uint32_t k = 64 * (1 + rng() % 272), m = 1 + rng() % (i % 2 ? 20000 : 4000), n = 1 + rng() % 1000;
        const size_t mem = i % 5 ? (size_t)64 << 20 : 0;
        const GemmPlan p = gemm_tc_search(ty, k, m, n, xdt, 148, mem, room), q = gemm_tc_search(ty, k, m, n, xdt, 148, mem, none), r = gemm_tc_search(ty, k, m, n, xdt, 148, mem);
        bad += q.cluster || r.cluster || q.tok != r.tok || q.dealt != r.dealt || q.waves != r.waves || q.nacc != r.nacc;
        if (!p.cluster) { bad += p.tok != r.tok || p.dealt != r.dealt || p.waves != r.waves || p.nacc != r.nacc; continue; }
        const uint32_t items = (m + 127) / 128 * ((n + p.tok - 1) / p.tok), units = (k + 255) / 256;
        bad += p.tok == 0 || p.tok % 16 || p.tok > 256 || p.dealt || p.waves || p.floats || items > room[p.cluster] || units < 2 * p.cluster || xdt == DT_F32;
        const uint32_t last = units / p.cluster * 4 - 3;  // k-blocks of the shortest part at least: every accumulator gets one
        bad += (p.chains != 1 && p.chains != 2 && p.chains != 4) || p.chains * p.tok > 256 || last < p.chains;
        accs |= p.chains;
        sizes |= 1u << p.cluster;
    }
    printf("%u %u %u\n", bad, sizes, accs);
}
"""


def test_plans_with_clusters(tmp_path):
    (tmp_path / "model.cu").write_text(MODEL)
    subprocess.run([build.nvcc(), "-O2", "-std=c++17", *build.ARCH, "-I", str(build.CSRC), str(tmp_path / "model.cu"), "-o", str(tmp_path / "model")], check=True)
    bad, sizes, accs = map(int, subprocess.run([str(tmp_path / "model")], check=True, capture_output=True, text=True).stdout.split())
    assert bad == 0 and sizes == 0b101111100 | sizes & 0b10000000 and accs == 7
