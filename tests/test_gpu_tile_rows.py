"""The tensor-core matmul's ways of bringing blocks as stored into shared memory, at their edges: row pitches that make a
tensor map of one, two, four or eight rows (every number of blocks to a row modulo eight), heights that such groups of rows divide
and heights that they do not, tensors on 2-byte boundaries, rows that end inside a unit of 256 weights, and token counts at the
edges of sixteens, of one and two accumulators (128) and of items (256)."""
import numpy as np
import pytest
import torch

from chatokf_b200 import synth
from chatokf_b200.enc import CudaEnc, GGUFTensor
from chatokf_b200.gguf_types import GGUFType, block_elems
from helpers import rel_err

pytestmark = pytest.mark.gpu

# both operands rounded once, 2^-12 (fp16) or 2^-9 (bf16) each at most, products' errors like a random walk: below twice that
TOL = {torch.float16: 1e-3, torch.bfloat16: 8e-3}
# (units to a row, rows, tokens)
SHAPES = [(1, 136, 9), (2, 136, 16), (3, 131, 17), (4, 260, 128), (5, 8, 129), (7, 129, 130), (8, 131, 64), (9, 1, 33), (20, 264, 256),
          (6, 1032, 257), (2, 4000, 300)]


@pytest.mark.parametrize("ty", list(GGUFType))
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
def test_rows_of_every_pitch(ctx, ty, dt):
    for i, (units, m, n) in enumerate(SHAPES):
        k = units * 256
        if block_elems(ty) < 256 and i % 2:  # a last unit of 64 or 128 weights
            k -= 256 - max(64, block_elems(ty))
        woff = 0 if i % 3 else 16 if ty == GGUFType.Q4_K else 2 * (i + 1)
        rng = np.random.default_rng(100 * i + int(ty))
        blocks = synth.random_blocks(ty, m * k // block_elems(ty), rng)
        w = ctx.upload(np.concatenate([np.zeros(woff, np.uint8), blocks]))
        t = GGUFTensor("w", (k, m), ty, woff)
        X = torch.from_numpy(rng.normal(size=(n, k)).astype(np.float32)).cuda().to(dt)
        enc, want = CudaEnc(ctx), torch.empty(n, m, device="cuda")
        ctx.set_flags(1)
        try:
            enc.gemm(t, X, want, w, n)
        finally:
            ctx.set_flags(0)
        got = torch.full((n * m + 8,), float("nan"), device="cuda")
        before = ctx.fallbacks
        enc.gemm(t, X, got, w, n)
        torch.cuda.synchronize()
        assert ctx.fallbacks == before and ctx.device_status() == 0
        assert torch.isnan(got[n * m:]).all(), "wrote past the N * M outputs"
        assert rel_err(got[:n * m].reshape(n, m).cpu().numpy(), want.cpu().numpy()) <= TOL[dt], (k, m, n, woff)
