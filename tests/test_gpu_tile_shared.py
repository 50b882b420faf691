"""Prefill matmuls whose items are shared by clusters of CTAs along K, against the plain kernels: every cluster size, parts of different
length, a last unit that is not whole, heights and outputs that leave results off 16 bytes, tokens around the multiples of 16, both kinds of
outputs, weights that arrive by plain copies; the same bits from a second call, nothing written past the outputs; inside a graph and without
working memory."""
import numpy as np
import pytest
import torch

from chatokf_b200 import synth
from chatokf_b200.enc import CudaEnc, GGUFTensor
from chatokf_b200.gguf_types import GGUFType, block_elems, row_byte_count

pytestmark = pytest.mark.gpu

# k, m, n: few enough 128-row items for clusters of 2 (74 of them) to 8 (15)
SHAPES = [(1280, 4000, 20), (1600, 5000, 33), (2112, 3001, 16), (4096, 1500, 34), (4672, 130, 97), (8192, 1023, 9), (2816, 515, 240), (6144, 2048, 500), (17408, 258, 70),
          (8960, 8385, 19), (9984, 295, 1020)]


@pytest.mark.parametrize("ty", list(GGUFType))
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16, torch.float32])
def test_shared_items(ctx, ty, dt):
    enc = CudaEnc(ctx)
    pool = torch.from_numpy(synth.random_blocks(ty, 4096, np.random.default_rng(2)).reshape(4096, -1)).cuda()
    for i, (k, m, n) in enumerate(SHAPES):
        k = k // max(64, block_elems(ty)) * max(64, block_elems(ty))
        gen = torch.Generator("cuda").manual_seed(k + n)
        count, shift = k // block_elems(ty) * m, (0 if ty == GGUFType.Q4_K or i % 3 else 2)
        buf = torch.zeros(count * pool.shape[1] + 258, dtype=torch.uint8, device="cuda")
        buf[shift:shift + count * pool.shape[1]] = pool[torch.randint(0, 4096, (count,), device="cuda", generator=gen)].view(-1)
        w, t = ctx.wrap(buf, count * pool.shape[1] + shift), GGUFTensor("w", (k, m), ty, shift)
        X = torch.randn(n, k, device="cuda", generator=gen).to(dt)
        odt, first = [torch.float32, torch.bfloat16][i % 2], [0, 0, 1][i % 3]
        want = torch.empty(n, m, device="cuda")
        ctx.set_flags(1)
        try:
            enc.gemm(t, X, want, w, n)
        finally:
            ctx.set_flags(0)
        outs = []
        for _ in range(2):
            full = torch.full((first + n * m + 8,), float("nan"), device="cuda", dtype=odt)
            enc.gemm(t, X, full[first:first + n * m], w, n)
            outs.append(full)
        torch.cuda.synchronize()
        assert torch.isnan(outs[0][:first]).all() and torch.isnan(outs[0][first + n * m:]).all()
        got = outs[0][first:first + n * m].view(n, m)
        assert torch.equal(got, outs[1][first:first + n * m].view(n, m))
        # both operands rounded once, to fp16 (2^-11) or bf16 (2^-8), K terms of random sign: a few of these steps of max|y|; a bf16 result half a step more
        tol = (2e-3 if dt == torch.float16 else 1e-2) + (4e-3 if odt == torch.bfloat16 else 0)
        assert float((got.float() - want).abs().max() / want.abs().max()) <= tol, (k, m, n)
    assert ctx.device_status() == 0


def test_shared_items_in_a_graph_and_without_working_memory(ctx):
    k, m, n = 9728, 2560, 77
    w = ctx.upload(synth.random_blocks(GGUFType.Q4_K, m * k // 256, np.random.default_rng(4)))
    t, enc = GGUFTensor("w", (k, m), GGUFType.Q4_K), CudaEnc(ctx)
    x, out, other = torch.randn(n, k, device="cuda").bfloat16(), torch.zeros(n, m, device="cuda"), torch.zeros(n, m, device="cuda")
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        enc.gemm(t, x, out, w, n)
        want = out.clone()
        out.zero_()
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            enc.gemm(t, x, out, w, n)
            enc.gemm(t, x, out, w, n)
        g.replay()
        enc.gemm_noalloc(t, x, other, w, n)
    torch.cuda.synchronize()
    assert torch.equal(out, want) and torch.equal(other, want)
    assert ctx.device_status() == 0
