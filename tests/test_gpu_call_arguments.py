"""What the operators read out of torch's objects: plain tensors, parameters and other subclasses, tensors without an address, other things;
and the stream that is current where the call is made."""
import numpy as np
import pytest
import torch

from chatokf_b200 import synth
from chatokf_b200.enc import CudaEnc, GGUFTensor
from chatokf_b200.gguf_types import GGUFType

pytestmark = pytest.mark.gpu


@pytest.fixture()
def problem(ctx):
    k, m = 512, 64
    w = ctx.upload(synth.random_blocks(GGUFType.Q8_0, m * k // 32, np.random.default_rng(1)))
    x = torch.randn(k, device="cuda").half()
    want = torch.empty(m, device="cuda")
    t, enc = GGUFTensor("w", (k, m), GGUFType.Q8_0), CudaEnc(ctx)
    enc.gemm(t, x, want, w, 1)
    torch.cuda.synchronize()
    return enc, t, w, x, want


def test_kinds_of_tensors(problem):
    enc, t, w, x, want = problem

    class Named(torch.Tensor):
        pass

    for X in (torch.nn.Parameter(x, requires_grad=False), x.as_subclass(Named), torch.stack([x, x])[1], x.float().requires_grad_()):
        out = torch.empty(t.M, device="cuda")
        enc.gemm(t, X, out.as_subclass(Named), w, 1)
        torch.cuda.synchronize()
        assert torch.equal(out, want)


def test_what_has_no_address_or_type_raises(problem):
    enc, t, w, x, want = problem
    out = torch.empty(t.M, device="cuda")
    with pytest.raises(KeyError):
        enc.gemm(t, x.double(), out, w, 1)
    with pytest.raises(AttributeError):
        enc.gemm(t, np.zeros(t.K, np.float32), out, w, 1)
    with pytest.raises(RuntimeError):
        torch.vmap(lambda v: (enc.gemm(t, v, out, w, 1), v)[1])(torch.stack([x, x]))
    enc.gemm(t, x, out, w, 1)  # still works
    torch.cuda.synchronize()
    assert torch.equal(out, want)


def test_current_stream(problem):
    enc, t, w, x, want = problem
    s, out, late = torch.cuda.Stream(), torch.zeros(t.M, device="cuda"), torch.zeros_like(x)
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        torch.cuda._sleep(20_000_000)  # about 10 ms
        late.copy_(x)
        enc.gemm(t, late, out, w, 1)
    s.synchronize()
    assert torch.equal(out, want)
