"""The tensor-core matmul's working memory (bf16 copies of fp32 activations, partial tiles): one set per
stream, one per graph.  A replay must not depend on what other calls of the context do with theirs."""
import gc

import numpy as np
import pytest
import torch

from chatokf_b200 import synth
from chatokf_b200.enc import Context, CudaEnc, GGUFTensor
from chatokf_b200.gguf_types import GGUFType, block_elems
from helpers import rel_err

pytestmark = pytest.mark.gpu

K, M = 4096, 1000  # eight slabs: dealt out at every token count below 512


@pytest.fixture()
def own(lib_built):
    c = Context(0)
    w = c.upload(synth.random_blocks(GGUFType.Q4_0, M * K // block_elems(GGUFType.Q4_0), np.random.default_rng(4)))
    yield c, w, GGUFTensor("w", (K, M), GGUFType.Q4_0)
    torch.cuda.synchronize()
    c.close()


def launches(c, f):
    before = c.launches
    f()
    return c.launches - before


@pytest.mark.parametrize("warm", [False, True])
@pytest.mark.parametrize("same", [False, True])
def test_a_replay_after_larger_calls(own, warm, same):
    """Captured on the stream that the context has worked on or on a fresh one, with and without a call before;
    then larger calls, for which the stream's buffers are replaced; then the replay."""
    c, w, t = own
    a = torch.cuda.Stream()
    b = a if same else torch.cuda.Stream()
    n, big = 40, 700
    X, Y = torch.randn(n, K, device="cuda"), torch.randn(big, K, device="cuda")
    want, got = torch.empty(n, M, device="cuda"), torch.empty(n, M, device="cuda")
    other = torch.empty(big, M, device="cuda")
    CudaEnc(c, torch.cuda.Stream()).gemm(t, X, want, w, n)
    if warm:
        CudaEnc(c, a).gemm(t, X, got, w, n)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=b):
        taken = launches(c, lambda: CudaEnc(c, torch.cuda.current_stream()).gemm(t, X, got, w, n))
        if not same:  # a call beside the capture, on a stream that it does not touch
            CudaEnc(c, a).gemm(t, Y[:300], other, w, 300)
    assert taken == 3, "converted once, dealt out, summed"
    for _ in range(3):
        got.zero_()
        torch.cuda.synchronize()
        CudaEnc(c, a).gemm(t, Y, other, w, big)
        with torch.cuda.stream(b):
            g.replay()
        torch.cuda.synchronize()
        assert torch.equal(got, want)
    assert c.device_status() == 0


def test_replays_beside_calls_and_other_replays(own):
    """Two graphs captured one after the other on one stream, replayed on streams of their own beside calls on a third."""
    c, w, t = own
    n = 40
    X = [torch.randn(n, K, device="cuda") for _ in range(3)]
    want, got = [[torch.empty(n, M, device="cuda") for _ in X] for _ in range(2)]
    streams = [torch.cuda.Stream() for _ in X]
    for x, o in zip(X, want):
        CudaEnc(c, streams[0]).gemm(t, x, o, w, n)
    torch.cuda.synchronize()
    graphs = []
    for x, o in zip(X[:2], got):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=streams[0]):
            CudaEnc(c, torch.cuda.current_stream()).gemm(t, x, o, w, n)
        graphs.append(g)
    torch.cuda.synchronize()
    for _ in range(30):
        for g, s in zip(graphs, streams):
            with torch.cuda.stream(s):
                g.replay()
        CudaEnc(c, streams[2]).gemm(t, X[2], got[2], w, n)
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    assert c.device_status() == 0


def test_a_graphs_memory_is_given_back(own):
    c, w, t = own
    n = 8192  # 64 MiB of bf16 activations
    X, out = torch.randn(n, K, device="cuda"), torch.empty(n, M, device="cuda")
    enc = CudaEnc(c)
    enc.gemm(t, X, out, w, n)
    torch.cuda.synchronize()

    def used():
        torch.cuda.synchronize()
        free, total = torch.cuda.mem_get_info()
        return total - free

    graphs = []
    for _ in range(8):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            CudaEnc(c, torch.cuda.current_stream()).gemm(t, X, out, w, n)
        graphs.append(g)
    held = used()
    del g
    graphs.clear()
    gc.collect()
    torch.cuda.synchronize()
    enc.gemm(t, X, out, w, n)  # a call outside captures frees what no graph holds
    assert held - used() >= 8 * (60 << 20)


def test_more_streams_than_sets(own):
    """Sixteen streams have a set each; further ones convert in the tile and deal nothing out, until a set
    has been idle for 1024 matmuls."""
    c, w, t = own
    n = 40
    X, want, got = torch.randn(n, K, device="cuda"), torch.empty(n, M, device="cuda"), torch.empty(n, M, device="cuda")
    streams = [torch.cuda.Stream() for _ in range(20)]
    ids = {s.cuda_stream for s in streams}
    assert len(ids) == 20
    for i, s in enumerate(streams):
        assert launches(c, lambda: CudaEnc(c, s).gemm(t, X, got, w, n)) == (3 if i < 16 else 1)
        torch.cuda.synchronize()
        if i == 0:
            want.copy_(got)
        # the same operands, fp32 sums in another order
        assert rel_err(got.cpu().numpy(), want.cpu().numpy()) <= 1e-5
    for _ in range(1024):
        CudaEnc(c, streams[0]).gemm(t, X, got, w, n)
    assert launches(c, lambda: CudaEnc(c, streams[19]).gemm(t, X, got, w, n)) == 3
    assert launches(c, lambda: CudaEnc(c, streams[0]).gemm(t, X, got, w, n)) == 3
    torch.cuda.synchronize()
    assert torch.equal(got, want)
    assert c.device_status() == 0


def test_more_activations_than_a_set_keeps(lib_built):
    """256 MiB of bf16 activations are kept at most: more are converted and multiplied run by run of tokens."""
    c = Context(0)
    k, m, n = 17408, 70, 8201
    w = c.upload(synth.random_blocks(GGUFType.Q4_0, m * k // 32, np.random.default_rng(5)))
    t = GGUFTensor("w", (k, m), GGUFType.Q4_0)
    X = torch.randn(n, k, device="cuda")
    got, want = torch.full((n * m + 8,), float("nan"), device="cuda"), torch.empty(n * m, device="cuda")
    CudaEnc(c).gemm(t, X.bfloat16(), want, w, n)
    CudaEnc(c).gemm(t, X, got, w, n)
    torch.cuda.synchronize()
    assert torch.isnan(got[n * m:]).all()
    # the same operands, fp32 sums in another order
    assert rel_err(got[:n * m].cpu().numpy(), want.cpu().numpy()) <= 1e-5
    assert c.device_status() == 0
    c.close()
