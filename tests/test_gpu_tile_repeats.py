"""The tensor-core matmul sums in one order whatever the timing, so the same call gives the same bits every time.  Weights come from
HBM (copies of the same bytes that together exceed L2, taken in turn), so that what a ring holds lands at all sorts of times."""
import numpy as np
import pytest
import torch

from chatokf_b200 import synth
from chatokf_b200.enc import CudaEnc, GGUFTensor
from chatokf_b200.gguf_types import GGUFType, block_elems, row_byte_count
from helpers import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ty", list(GGUFType))
@pytest.mark.parametrize("dt,odt", [(torch.float16, torch.bfloat16), (torch.bfloat16, torch.float32)])
@pytest.mark.parametrize("k,m,woff", [(2048, 5000, 0), (4096, 5000, 0), (4160, 4999, 2)])
def test_same_bits_every_time(ctx, ty, dt, odt, k, m, woff):
    """Whole and dealt items of 16 to 256 tokens, which set the depth of the rings; tensors that tensor maps describe and,
    with a row length and an offset that they cannot, tensors that come by other copies (Q4_K: always on 16 bytes)."""
    k = k // block_elems(ty) * block_elems(ty)
    woff = 16 * (woff > 0) if ty == GGUFType.Q4_K else woff
    size = row_byte_count(ty, k) * m
    stride = (woff + size + 255) // 256 * 256
    copies = (160 << 20) // stride + 1
    blocks = synth.random_blocks(ty, m * k // block_elems(ty), np.random.default_rng(int(ty)))
    data = torch.zeros(copies * stride + 256, dtype=torch.uint8, device="cuda")
    data[:copies * stride].view(copies, stride)[:, woff:woff + size] = torch.from_numpy(blocks).cuda()
    w = ctx.wrap(data, copies * stride)
    views = [GGUFTensor("w", (k, m), ty, c * stride + woff) for c in range(copies)]
    enc = CudaEnc(ctx)
    for n in (16, 64, 128, 240, 256, 700):
        X = torch.randn(n, k, device="cuda", generator=torch.Generator("cuda").manual_seed(n)).to(dt)
        want, got = torch.empty(n, m, device="cuda"), torch.empty(n, m, dtype=odt, device="cuda")
        ctx.set_flags(1)
        try:
            enc.gemm(views[0], X, want, w, n)
        finally:
            ctx.set_flags(0)
        bits = torch.int16 if odt == torch.bfloat16 else torch.int32
        first, same = None, torch.ones((), dtype=torch.bool, device="cuda")
        for i in range(30):
            got.fill_(float("nan"))
            enc.gemm(views[i % copies], X, got, w, n)
            first = got.clone() if first is None else first
            same &= (got.view(bits) == first.view(bits)).all()
        torch.cuda.synchronize()
        assert bool(same), n
        # both operands rounded once, 2^-12 or 2^-9 each at most, bf16 results another 2^-9 of their own size
        tol = {torch.float16: 1e-3, torch.bfloat16: 8e-3}[dt] + (4e-3 if odt == torch.bfloat16 else 0.0)
        assert rel_err(first.float().cpu().numpy(), want.cpu().numpy()) <= tol, n
    assert ctx.device_status() == 0
