"""The tensor-core matmul's unpacking, type by type, where it can go wrong: every quarter of a block (K of
one to five k-blocks and long), rows past the last slab, token counts around the sixteens that are staged,
tensors that start where only 2-byte loads are aligned.  Random blocks reach every code and scale."""
import numpy as np
import pytest
import torch

import oracle
from chatokf_b200 import synth
from chatokf_b200.enc import CudaEnc, GGUFTensor
from chatokf_b200.gguf_types import GGUFType, block_elems
from helpers import rel_err

pytestmark = pytest.mark.gpu

# both operands are rounded once: relative 2^-12 (fp16) or 2^-9 (bf16) each at most, and the products'
# errors add up like a random walk, so max|error| / max|y| stays below twice that
TOL = {torch.float16: 1e-3, torch.bfloat16: 8e-3, torch.float32: 8e-3}


@pytest.mark.parametrize("ty", list(GGUFType))
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16, torch.float32])
def test_tile_unpack(ctx, ty, dt):
    for k, m, n, woff in [(256, 1, 9, 0), (512, 129, 16, 32), (1280, 200, 17, 0), (4096, 140, 31, 0),
                          (2048, 70, 257, 16 if ty == GGUFType.Q4_K else 2)]:
        rng = np.random.default_rng(k + m + n)
        blocks = synth.random_blocks(ty, m * k // block_elems(ty), rng)
        w = ctx.upload(np.concatenate([np.zeros(woff, np.uint8), blocks]))
        X = torch.from_numpy(rng.normal(size=(n, k)).astype(np.float32)).cuda().to(dt)
        out = torch.full((n * m + 8,), float("nan"), device="cuda")
        before = ctx.fallbacks
        CudaEnc(ctx).gemm(GGUFTensor("w", (k, m), ty, woff), X, out, w, n)
        torch.cuda.synchronize()
        o = out.cpu().numpy()
        assert ctx.fallbacks == before
        assert np.isnan(o[n * m:]).all(), "wrote past the N * M outputs"
        want = oracle.matmul(ty, blocks, k, m, X.float().cpu().numpy(), n)
        assert rel_err(o[:n * m].reshape(n, m), want) <= TOL[dt], (k, m, n)
    assert ctx.device_status() == 0
