"""Two columns of long rows whose tiles are shared by clusters of two CTAs: heights just above one tile per SM and just below one and
a half, rows from 4 KB on, a last tile that is not whole, an odd number of units to a row (halves of different length), matrices
that share a launch."""
import numpy as np
import pytest
import torch

from chatokf_b200 import synth
from chatokf_b200.enc import CudaEnc, GGUFTensor
from chatokf_b200.gguf_types import GGUFType, block_elems, row_byte_count
from helpers import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ty", list(GGUFType))
@pytest.mark.parametrize("dt", [torch.float32, torch.float16])
def test_halved_tiles(ctx, ty, dt):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    units = -(-4096 // row_byte_count(ty, 256))
    for u, rows in [(units, [16 * sms + 1]), (units + 3, [24 * sms - 7]), (units | 1, [8 * sms, 12 * sms + 5])]:
        k, m = 256 * u, sum(rows)
        rng = np.random.default_rng(u + m)
        w = ctx.upload(synth.random_blocks(ty, m * k // block_elems(ty), rng))
        X = torch.from_numpy(rng.normal(size=(2, k)).astype(np.float32)).cuda().to(dt)
        at, ts = 0, []
        for r in rows:
            ts.append(GGUFTensor("w", (k, r), ty, at))
            at += row_byte_count(ty, k) * r
        if any(t.offset % 16 for t in ts):
            ts = ts[:1]  # matvecs take tensors on 16-byte boundaries
        enc, want, got = CudaEnc(ctx), [torch.empty(2, t.M, device="cuda") for t in ts], [torch.empty(2, t.M, device="cuda") for t in ts]
        ctx.set_flags(1)
        try:
            for t, o in zip(ts, want):
                enc.gemm(t, X, o, w, 2)
        finally:
            ctx.set_flags(0)
        with enc.parallel():
            for t, o in zip(ts, got):
                enc.gemm(t, X, o, w, 2)
        torch.cuda.synchronize()
        assert ctx.device_status() == 0
        for g, o in zip(got, want):  # x carries 16 bits: 2^-15 / sqrt(12) of a unit's largest per term
            assert rel_err(g.cpu().numpy(), o.cpu().numpy()) <= 1e-4, (k, rows)
