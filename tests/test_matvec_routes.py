"""Which of the two matvec kernels a launch takes and how it is split, on the host, for shapes whose times the comments of the rules give."""
import subprocess

from chatokf_b200 import build
from chatokf_b200.gguf_types import GGUFType

MODEL = r"""
#include <cstdio>
#include "okf_gemv_ring.h"
using namespace okf;
static const StreamRoom room = {{148, 74, 33, 15}, {296, 148, 71, 33}};
template <int TY> static StreamPlan plan(int mode, uint32_t nunit, uint32_t n, uint32_t tiles) {
    if (mode == M_SEP) return stream_launches<TY, M_SEP>(nunit, n, tiles, room);
    if (mode == M_W1) return stream_launches<TY, M_W1>(nunit, n, tiles, room);
    if (mode == M_W2) return stream_launches<TY, M_W2>(nunit, n, tiles, room);
    if constexpr (TY == T_Q8_0 || TY == T_Q4_0 || TY == T_IQ4_NL || TY == T_Q2_0)
        return mode == M_R3 ? stream_launches<TY, M_R3>(nunit, n, tiles, room) : stream_launches<TY, M_R4>(nunit, n, tiles, room);
    return {};
}
int main() {
    int ty;
    uint32_t k, m, n, take;
    while (scanf("%d %u %u %u", &ty, &k, &m, &n) == 4) {
        const int mode = gemv_mode(k, DT_F32, n, take);
        GemvArgs a = {};
        a.n = take; a.nunit = (k + 255) / 256; a.tiles = (m + 15) / 16; a.row_bytes = k / block_elems(ty) * block_bytes(ty);
        StreamPlan p = {};
        switch (ty) {
        case T_Q8_0: p = plan<T_Q8_0>(mode, a.nunit, take, a.tiles); break;
        case T_Q4_K: p = plan<T_Q4_K>(mode, a.nunit, take, a.tiles); break;
        case T_Q6_K: p = plan<T_Q6_K>(mode, a.nunit, take, a.tiles); break;
        case T_IQ4_NL: p = plan<T_IQ4_NL>(mode, a.nunit, take, a.tiles); break;
        case T_IQ2_XXS: p = plan<T_IQ2_XXS>(mode, a.nunit, take, a.tiles); break;
        }
        const bool stream = p.ok && p.us < ring_estimate(ty, mode, a, 148);
        printf("%d %u %u %d\n", stream, stream ? 1u << p.L.clog : 0, stream ? (a.tiles + p.tiles - 1) / p.tiles : 1, stream ? p.early : 1);
    }
}
"""
# type, k, m, columns: streaming kernel, CTAs of a cluster, launches, starts beside its predecessor
ROUTES = [
    (GGUFType.Q8_0, 2304, 2729, 1, (0, 0, 1, 1)),      # a tile to a CTA, two of them on some SMs
    (GGUFType.Q6_K, 3072, 27634, 1, (0, 0, 1, 1)),
    (GGUFType.Q4_K, 5120, 65536, 1, (0, 0, 1, 1)),     # whole rows by bulk copies
    (GGUFType.Q6_K, 2560, 151936, 1, (0, 0, 1, 1)),
    (GGUFType.Q4_K, 2560, 2 * 9728, 1, (1, 1, 1, 1)),
    (GGUFType.Q8_0, 14336, 4096, 4, (1, 8, 1, 1)),
    (GGUFType.Q8_0, 1536, 154809, 4, (0, 0, 1, 1)),    # x staged once for many tiles
    (GGUFType.IQ4_NL, 1024, 209, 8, (1, 1, 1, 1)),
    (GGUFType.IQ2_XXS, 23040, 64269, 8, (1, 4, 2, 1)),  # the sums of all tiles do not fit
    (GGUFType.Q8_0, 7904, 59634, 4, (0, 0, 1, 1)),     # nor here, where a row ends inside a unit
    (GGUFType.IQ2_XXS, 24320, 28385, 4, (1, 4, 1, 0)),  # needs every SM in large clusters
]


def test_routes(tmp_path):
    (tmp_path / "model.cu").write_text(MODEL)
    subprocess.run([build.nvcc(), "-O2", "-std=c++17", "--expt-relaxed-constexpr", *build.ARCH, "-I", str(build.CSRC), str(tmp_path / "model.cu"), "-o", str(tmp_path / "model")],
                   check=True)
    asked = "".join(f"{int(ty)} {k} {m} {n}\n" for ty, k, m, n, _ in ROUTES)
    out = subprocess.run([str(tmp_path / "model")], input=asked, check=True, capture_output=True, text=True).stdout.split("\n")
    for (ty, k, m, n, want), line in zip(ROUTES, out):
        assert tuple(map(int, line.split())) == want, (ty, k, m, n)
