"""Results of the several-column matvec around the sizes at which its plan changes: how much of the ring a
resident x leaves to one CTA (two CTAs share K instead), and three or four tiles per SM (two CTAs per SM)."""
import numpy as np
import pytest
import torch

from chatokf_b200 import synth
from chatokf_b200.enc import CudaEnc, GGUFTensor
from chatokf_b200.gguf_types import GGUFType, block_elems
from helpers import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ty,k,n", [(GGUFType.Q8_0, 17408, 2), (GGUFType.Q8_0, 8192, 4), (GGUFType.Q5_K, 9728, 3), (GGUFType.Q4_K, 2048, 8),
                                    (GGUFType.Q2_0, 5120, 5), (GGUFType.IQ2_XXS, 5120, 3), (GGUFType.Q4_0, 8224, 4)])
@pytest.mark.parametrize("m", [3 * 148 * 16 - 1, 3 * 148 * 16, 4 * 148 * 16 + 1])
def test_plans(ctx, ty, k, n, m):
    w = ctx.upload(synth.random_blocks(ty, m * k // block_elems(ty), np.random.default_rng(k)))
    t = GGUFTensor("w", (k, m), ty)
    X = torch.randn(n, k, device="cuda").half()
    got, want = torch.full((n * m + 4,), float("nan"), device="cuda"), torch.empty(n * m, device="cuda")
    CudaEnc(ctx).gemm(t, X, got, w, n)
    ctx.set_flags(1)
    try:
        CudaEnc(ctx).gemm(t, X, want, w, n)
    finally:
        ctx.set_flags(0)
    torch.cuda.synchronize()
    assert torch.isnan(got[n * m:]).all()
    assert rel_err(got[:n * m].cpu().numpy(), want.cpu().numpy()) <= 1e-4  # activations of 16 bits, as everywhere
    assert ctx.device_status() == 0
