"""Prefill matmuls whose items are shared by clusters of CTAs, against the plain kernels: for every type that shares items every size of cluster and
number of accumulators; the kernels are counted, so that no other path takes their place."""
import numpy as np
import pytest
import torch

from chatokf_b200 import synth
from chatokf_b200.enc import CudaEnc, GGUFTensor
from chatokf_b200.gguf_types import GGUFType, block_elems, row_byte_count

pytestmark = pytest.mark.gpu

TYPES = [t for t in GGUFType if t != GGUFType.Q4_0]  # (Q4_0: dealt items)
# k, m, n: which sizes of cluster and accumulators they come to is looked at in test_cluster_plans.py
SHAPES = [(1792, 140, 10), (2112, 3001, 16), (4096, 1500, 34), (4672, 130, 97), (8192, 1023, 9), (2816, 515, 240), (6144, 2048, 500),
          (8960, 8385, 19), (3328, 550, 11), (5888, 2772, 84), (4864, 137, 11), (4480, 196, 10)]


def shapes(ty):
    step = max(64, block_elems(ty))
    return [(k // step * step, m, n) for k, m, n in SHAPES]


@pytest.mark.parametrize("ty", TYPES)
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16, torch.float32])
def test_clusters(ctx, ty, dt):
    enc = CudaEnc(ctx)
    pool = torch.from_numpy(synth.random_blocks(ty, 4096, np.random.default_rng(2)).reshape(4096, -1)).cuda()
    for i, (k, m, n) in enumerate(shapes(ty)):
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
            before = ctx.launches
            enc.gemm(t, X, full[first:first + n * m], w, n)
            assert ctx.launches - before == (2 if dt == torch.float32 else 1), "converted or not, no second kernel that adds up"
            outs.append(full)
        torch.cuda.synchronize()
        assert torch.isnan(outs[0][:first]).all() and torch.isnan(outs[0][first + n * m:]).all()
        got = outs[0][first:first + n * m].view(n, m)
        assert torch.equal(got, outs[1][first:first + n * m].view(n, m))
        # both operands rounded once, to fp16 (2^-11) or bf16 (2^-8), K terms of random sign: a few of these steps of max|y|; a bf16 result half a step more
        tol = (2e-3 if dt == torch.float16 else 1e-2) + (4e-3 if odt == torch.bfloat16 else 0)
        assert float((got.float() - want).abs().max() / want.abs().max()) <= tol, (k, m, n)
    assert ctx.device_status() == 0
