"""Items dealt out along K with the types that share them between clusters where they can: told not to (flag 2), what test_gpu_tile_dealing.py and
test_gpu_tile_repeats.py look at holds for them too.  Two kernels a call, the second one adds the partial tiles up."""
import numpy as np
import pytest
import torch

from chatokf_b200 import synth
from chatokf_b200.enc import Context, CudaEnc, GGUFTensor
from chatokf_b200.gguf_types import GGUFType, block_elems
from helpers import rel_err
from test_gpu_tile_clusters import TYPES

pytestmark = pytest.mark.gpu


@pytest.fixture()
def own(lib_built):
    """A context with working memory for all streams here: a stream that finds none runs its items whole, its sums in another order."""
    c = Context(0)
    yield c
    torch.cuda.synchronize()
    c.close()


@pytest.mark.parametrize("ty", TYPES)
@pytest.mark.parametrize("k,m,n", [(8192, 131, 45), (4096, 1000, 40), (9728, 2560, 77), (6144, 2048, 240)])
def test_dealt_items(own, ty, k, m, n):
    """Against the plain kernels, with fp32 and bf16 results, every call the same bits and on streams of their own."""
    ctx = own
    w = ctx.upload(synth.random_blocks(ty, m * k // block_elems(ty), np.random.default_rng(int(ty))))
    t, enc = GGUFTensor("w", (k, m), ty), CudaEnc(ctx)
    X = [torch.randn(n, k, device="cuda", generator=torch.Generator("cuda").manual_seed(i)).half() for i in range(4)]
    plain = [torch.empty(n, m, device="cuda") for _ in X]
    ctx.set_flags(1)
    for x, o in zip(X, plain):
        enc.gemm(t, x, o, w, n)
    streams = [torch.cuda.Stream() for _ in X]
    ctx.set_flags(2)
    for odt in (torch.float32, torch.bfloat16):
        want, got = [torch.empty(n, m, dtype=odt, device="cuda") for _ in X], [torch.empty(n, m, dtype=odt, device="cuda") for _ in X]
        for x, o in zip(X, want):
            before = ctx.launches
            enc.gemm(t, x, o, w, n)
            assert ctx.launches - before == 2, "dealt out, summed"
        torch.cuda.synchronize()
        for _ in range(10):
            for s, x, o in zip(streams, X, got):
                CudaEnc(ctx, s).gemm(t, x, o, w, n)
        torch.cuda.synchronize()
        for a, b, o in zip(got, want, plain):
            assert torch.equal(a, b)
            # both operands rounded once, 2^-12 each at most, bf16 results another 2^-9 of their own size
            assert rel_err(b.float().cpu().numpy(), o.cpu().numpy()) <= 1e-3 + (4e-3 if odt == torch.bfloat16 else 0.0)
    assert ctx.device_status() == 0
