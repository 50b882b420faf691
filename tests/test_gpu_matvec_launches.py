"""Streaming matvecs of tall matrices in several launches, and the rounding of long ragged rows."""
import numpy as np
import pytest
import torch

from chatokf_b200 import synth
from chatokf_b200.enc import CudaEnc, GGUFTensor
from chatokf_b200.gguf_types import GGUFType, block_elems, row_byte_count
from helpers import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ty,k,rows,n", [(GGUFType.Q8_0, 105 * 256, [3000, 1483], 8), (GGUFType.Q8_0, 105 * 256, [17270], 4), (GGUFType.IQ2_XXS, 89 * 256, [40990], 8),
                                         (GGUFType.IQ4_NL, 105 * 256 - 32, [9200], 4)])
def test_tiles_of_several_launches(ctx, ty, k, rows, n):
    """Matrices so tall that the sums of a cluster's tiles do not fit beside x: two launches, the border between them inside a matrix."""
    pool = torch.from_numpy(synth.random_blocks(ty, 4096, np.random.default_rng(k)).reshape(4096, -1)).cuda()
    gen = torch.Generator("cuda").manual_seed(n)
    at, ts = 0, []
    for m in rows:
        ts.append(GGUFTensor("w", (k, m), ty, at))
        at += (row_byte_count(ty, k) * m + 15) // 16 * 16
    buf = torch.zeros(at + 256, dtype=torch.uint8, device="cuda")
    for t in ts:
        count = k // block_elems(ty) * t.M
        buf[t.offset:t.offset + count * pool.shape[1]] = pool[torch.randint(0, 4096, (count,), device="cuda", generator=gen)].view(-1)
    w, X, enc = ctx.wrap(buf, at), torch.randn(n, k, device="cuda", generator=gen), CudaEnc(ctx)
    X = X.half() if k % 256 == 0 else X
    want, got = [torch.empty(n * t.M, device="cuda") for t in ts], [torch.full((n * t.M + 4,), float("nan"), device="cuda") for t in ts]
    ctx.set_flags(1)
    try:
        for t, o in zip(ts, want):
            enc.gemm(t, X, o, w, n)
    finally:
        ctx.set_flags(0)
    before = ctx.launches
    with enc.parallel():
        for t, o in zip(ts, got):
            enc.gemm(t, X, o, w, n)
    launched = ctx.launches - before
    torch.cuda.synchronize()
    assert launched >= 2 and ctx.device_status() == 0
    for t, o, g in zip(ts, want, got):
        assert torch.isnan(g[n * t.M:]).all()
        # x carries 16 bits, as above (ragged rows: as it is)
        assert rel_err(g[:n * t.M].cpu().numpy(), o.cpu().numpy()) <= 1e-4


def test_sums_of_long_ragged_rows(ctx):
    """Rows that end inside a unit have x as it is, what is left is the rounding of fp32 sums.  An addition rounds by some 2^-24 / sqrt(6) of what it gives, and m of
    them, of terms of random sign, end sqrt(m / 2) such roundings off: two blocks a unit in runs of four, then up to 17 runs, 0.86e-7 (0.83e-7 measured);
    all of a warp's 34 to 67 units in one run 1.1e-7 (measured)."""
    ty, k, m = GGUFType.Q2_0, 17280, 20000
    pool = torch.from_numpy(synth.random_blocks(ty, 4096, np.random.default_rng(int(ty))).reshape(4096, -1)).cuda()
    gen = torch.Generator("cuda").manual_seed(9)
    count = k // block_elems(ty) * m
    buf = torch.zeros(count * pool.shape[1] + 256, dtype=torch.uint8, device="cuda")
    buf[:count * pool.shape[1]] = pool[torch.randint(0, 4096, (count,), device="cuda", generator=gen)].view(-1)
    w, t, enc = ctx.wrap(buf, count * pool.shape[1]), GGUFTensor("w", (k, m), ty), CudaEnc(ctx)
    X, out, W = torch.randn(1, k, device="cuda", generator=gen), torch.empty(1, m, device="cuda"), torch.empty(m * k, device="cuda")
    enc.gemm(t, X, out, w, 1)
    enc.dequantRow(w, W, m * k, ty, 0)
    want = torch.cat([X.double() @ a.double().T for a in W.view(m, k).split(1000)], 1)
    rms = float((out.double() - want).pow(2).mean().sqrt() / want.pow(2).mean().sqrt())
    assert rms <= 9.5e-8
    assert ctx.device_status() == 0
