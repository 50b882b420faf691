"""The host operator looks at all of a buffer before kernels address it: page-locked at its first byte only, or
in two registrations; and memory that is not the CPU's goes through the copy engine, as it always did."""
import mmap

import numpy as np
import pytest
import torch

from chatokf_b200 import synth
from chatokf_b200.enc import GGUFTensor, OkfError, QB
from chatokf_b200.gguf_types import GGUFType

pytestmark = pytest.mark.gpu

K, M, N = 4096, 3000, 2  # x of eight pages, out of six
PAGE = mmap.PAGESIZE


@pytest.fixture()
def case(ctx):
    w = ctx.upload(synth.random_blocks(GGUFType.Q8_0, K * M // 32, np.random.default_rng(1)))
    t = GGUFTensor("w", (K, M), GGUFType.Q8_0)
    x = np.random.default_rng(2).normal(size=(N, K)).astype(np.float32)
    return QB(ctx), w, t, x, QB(ctx).matmul(t, w, x, N)


@pytest.mark.parametrize("locked", [[(0, 1)], [(0, 3), (3, 2)], [(0, 2), (7, 1)], [(0, 16)], [(1, 15)]])
def test_partly_page_locked(ctx, case, locked):
    """`locked`: registered ranges as (first page, pages) of the sixteen that x and out are laid in."""
    qb, w, t, x, want = case
    bufs = [np.frombuffer(mmap.mmap(-1, 16 * PAGE), np.float32) for _ in range(2)]
    rt = torch.cuda.cudart()
    for b in bufs:
        for first, pages in locked:
            assert int(rt.cudaHostRegister(b.ctypes.data + first * PAGE, pages * PAGE, 0)) == 0
    try:
        for shift in (0, 4, 5):  # 16-byte aligned, and not
            X, out = bufs[0][shift:shift + N * K].reshape(N, K), bufs[1][shift:shift + N * M].reshape(N, M)
            X[:] = x
            out[:] = np.nan
            qb.matmul(t, w, X, N, out)
            assert np.array_equal(out, want)
    finally:
        for b in bufs:
            for first, _ in locked:
                rt.cudaHostUnregister(b.ctypes.data + first * PAGE)


def test_device_memory(ctx, case):
    """Device pointers are no host buffers; the copy engine takes or refuses them, and nothing is touched by the CPU."""
    qb, w, t, x, want = case
    X, out = torch.from_numpy(x).cuda(), torch.zeros(N, M, device="cuda")
    try:
        qb.matmul_at(t, w, X.data_ptr(), N, out.data_ptr())
    except OkfError:
        pass
    else:
        assert np.array_equal(out.cpu().numpy(), want)
    assert np.array_equal(qb.matmul(t, w, x, N), want)
