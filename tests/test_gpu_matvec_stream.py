"""The streaming matvec where its split changes: fewer units than warps, borders of warps inside tiles and on them, K cut between clusters into
slices of different length, heights that are no multiple of a tile in matrices that share a launch, as many tiles as one wave has room for and one
more, rows on every 2-byte offset its type allows; and that a call gives the same bits again."""
import numpy as np
import pytest
import torch

from chatokf_b200 import synth
from chatokf_b200.enc import CudaEnc, GGUFTensor
from chatokf_b200.gguf_types import GGUFType, block_elems, row_byte_count
from helpers import rel_err

pytestmark = pytest.mark.gpu

# x carries 16 bits: 2^-15 / sqrt(12) of a unit's largest per term, 1e-4 of max|y| as in every matvec test
SHAPES = [(256, [16]), (512, [40]), (768, [7, 129]), (1280, [148 * 16, 16]), (2304, [149 * 16]), (2560, [300, 5000, 33]), (4864, [297 * 16 - 3]),
          (6400, [1]), (9728, [2560]), (11008, [923, 60]), (17408, [2600])]


@pytest.mark.parametrize("ty", list(GGUFType))
@pytest.mark.parametrize("n", [1, 2, 4, 5, 8])
def test_split(ctx, ty, n):
    for i, (k, rows) in enumerate(SHAPES):
        if i % 2 and block_elems(ty) < 256 and n < 5:
            k -= block_elems(ty)  # rows that end inside a unit: matrices leave one by one
        dt = [torch.float32, torch.float16, torch.bfloat16][(i + n) % 3]
        at, ts = 0, []
        for m in rows:
            ts.append(GGUFTensor("w", (k, m), ty, at))
            at += (row_byte_count(ty, k) * m + 15) // 16 * 16
        blocks = synth.random_blocks(ty, 4096, np.random.default_rng(k))
        pool = torch.from_numpy(blocks.reshape(4096, -1)).cuda()
        buf = torch.zeros(at + 256, dtype=torch.uint8, device="cuda")
        gen = torch.Generator("cuda").manual_seed(k + n)
        for t in ts:
            count = k // block_elems(ty) * t.M
            pick = torch.randint(0, 4096, (count,), device="cuda", generator=gen)
            buf[t.offset:t.offset + count * pool.shape[1]] = pool[pick].view(-1)
        w, X, enc = ctx.wrap(buf, at), torch.randn(n, k, device="cuda", generator=gen).to(dt), CudaEnc(ctx)
        want = [torch.empty(n * t.M, device="cuda") for t in ts]
        ctx.set_flags(1)
        try:
            for t, o in zip(ts, want):
                enc.gemm(t, X, o, w, n)
        finally:
            ctx.set_flags(0)
        runs = []
        for _ in range(2):
            got = [torch.full((n * t.M + 4,), float("nan"), device="cuda") for t in ts]
            with enc.parallel():
                for t, o in zip(ts, got):
                    enc.gemm(t, X, o, w, n)
            runs.append(got)
        torch.cuda.synchronize()
        top = max(float(o.abs().max()) for o in want)  # (a single row may sum to next to nothing)
        for t, o, a, b in zip(ts, want, *runs):
            assert torch.isnan(a[n * t.M:]).all(), "wrote past the N * M outputs"
            assert torch.equal(a[:n * t.M], b[:n * t.M])
            if n * t.M >= 64:
                assert rel_err(a[:n * t.M].cpu().numpy(), o.cpu().numpy()) <= 1e-4, (k, t.M)
            else:
                assert float((a[:n * t.M] - o).abs().max()) <= 1e-3 * top, (k, t.M)
    assert ctx.device_status() == 0


@pytest.mark.parametrize("n", [1, 3, 8])
def test_no_bytes_behind_the_last_block_are_taken_for_weights(ctx, n):
    """The last row of the last tile against bytes behind it that read as infinite scales."""
    for ty in GGUFType:
        k, m = 2048 + (256 if block_elems(ty) == 256 else block_elems(ty)), 37
        size = row_byte_count(ty, k) * m
        buf = torch.full((size + 256,), 0x7C, dtype=torch.uint8, device="cuda")
        buf[:size] = torch.from_numpy(synth.random_blocks(ty, m * k // block_elems(ty), np.random.default_rng(1)).reshape(-1)).cuda()
        X, out, want = torch.randn(n, k, device="cuda").half(), torch.empty(n * m, device="cuda"), torch.empty(n * m, device="cuda")
        w, t, enc = ctx.wrap(buf, size), GGUFTensor("w", (k, m), ty), CudaEnc(ctx)
        enc.gemm(t, X, out, w, n)
        ctx.set_flags(1)
        try:
            enc.gemm(t, X, want, w, n)
        finally:
            ctx.set_flags(0)
        torch.cuda.synchronize()
        assert rel_err(out.cpu().numpy(), want.cpu().numpy()) <= 1e-4, ty
    assert ctx.device_status() == 0
