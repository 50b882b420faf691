"""The several-column matvec kernels at the edges of their ranges, against the CPU oracle: one and two
sets of byte columns, K split over clusters of CTAs, rows that are no multiple of 256 weights."""
import numpy as np
import pytest
import torch

import oracle
from chatokf_b200 import synth
from chatokf_b200.enc import CudaEnc, GGUFTensor
from chatokf_b200.gguf_types import GGUFType, block_elems
from helpers import rel_err

pytestmark = pytest.mark.gpu

DTS = [torch.float32, torch.float16, torch.bfloat16]
# activations carry 16 bits relative to the largest of 256: a step of 2^-15 of that, an rms error of
# 2^-15 / sqrt(12) of it per term; 1e-4 of max|y| is the bound of every matvec test here
WIDE_TOL = 1e-4
# x as it is: what is left is the rounding of the oracle's own sequential
# fp32 sum of K terms (about sqrt(K) * 2^-24 of max|y|, 8e-6 at K = 16384)
RAGGED_TOL = 1e-5


def run(ctx, ty, k, m, n, dt, seed=0):
    rng = np.random.default_rng(k + m + seed)
    blocks = synth.random_blocks(ty, m * k // block_elems(ty), rng)
    w = ctx.upload(blocks)
    X = torch.from_numpy(rng.normal(size=(n, k)).astype(np.float32)).cuda().to(dt)
    out = torch.full((n * m + 4,), float("nan"), device="cuda")
    CudaEnc(ctx).gemm(GGUFTensor("w", (k, m), ty), X, out, w, n)
    torch.cuda.synchronize()
    o = out.cpu().numpy()
    assert np.isnan(o[n * m:]).all(), "wrote past the N * M outputs"
    return rel_err(o[:n * m].reshape(n, m), oracle.matmul(ty, blocks, k, m, X.float().cpu().numpy(), n))


@pytest.mark.parametrize("ty", list(GGUFType))
@pytest.mark.parametrize("n", [2, 4, 5, 8])
def test_columns(ctx, ty, n):
    """One unit, odd heights, rows long enough for clusters of two and four CTAs (the last with units
    that do not divide), several groups of tiles per CTA."""
    for i, (k, m) in enumerate([(256, 1), (1024, 33), (2560, 20011), (9728, 300), (17408, 100), (13056, 1300)]):
        assert run(ctx, ty, k, m, n, DTS[(i + n) % 3]) <= WIDE_TOL, (k, m)
    assert ctx.device_status() == 0


@pytest.mark.parametrize("ty", list(GGUFType))
def test_one_column_of_long_rows(ctx, ty):
    """Some more tiles than two to an SM (148 SMs), each halved between two CTAs: an odd number of units, a last
    tile of one row; and one tile fewer, which is not halved."""
    for k, m in [(10496, 296 * 16 + 1), (10496, 296 * 16)]:
        assert run(ctx, ty, k, m, 1, torch.float16, seed=2) <= WIDE_TOL, (k, m)
    assert ctx.device_status() == 0


@pytest.mark.parametrize("ty", [GGUFType.Q8_0, GGUFType.Q4_0, GGUFType.IQ4_NL, GGUFType.Q2_0])
@pytest.mark.parametrize("n", [1, 3, 4, 5, 8, 13])
def test_rows_that_end_inside_a_unit(ctx, ty, n):
    """From one block to several chunks, first and last block of a unit, four columns and a
    remainder, and the passes over a few tokens more than eight that K not a multiple of 64 takes."""
    step = block_elems(ty)
    for i, (k, m) in enumerate([(step, 5), (256 + step, 16), (1024 - step, 77), (4096 + step, 1000), (16384 - step, 40)]):
        if n > 8 and k % 64 == 0:
            continue  # the tensor-core tile, with 16-bit operands
        assert run(ctx, ty, k, m, n, DTS[(i + n) % 3], seed=1) <= RAGGED_TOL, (k, m)
    assert ctx.device_status() == 0


def test_the_next_rows_scales_stay_out(ctx):
    """The bytes behind a row's last block are the next row's: an infinite scale there meets zeros of x."""
    k, m = 288, 3
    blocks = synth.random_blocks(GGUFType.Q8_0, m * k // 32, np.random.default_rng(3))
    blocks.reshape(-1, 34)[9, :2] = np.frombuffer(np.float16(np.inf).tobytes(), np.uint8)  # row 1, block 0
    w = ctx.upload(blocks)
    x = torch.ones(k, device="cuda")
    out = torch.zeros(m, device="cuda")
    CudaEnc(ctx).gemm(GGUFTensor("w", (k, m), GGUFType.Q8_0), x, out, w, 1)
    torch.cuda.synchronize()
    o, want = out.cpu().numpy(), oracle.matvec(GGUFType.Q8_0, blocks, k, m, np.ones(k, np.float32))
    assert not np.isfinite(o[1]) and rel_err(o[[0, 2]], want[[0, 2]]) <= RAGGED_TOL


RAGGED = [GGUFType.Q8_0, GGUFType.Q4_0, GGUFType.IQ4_NL, GGUFType.Q2_0]


@pytest.mark.parametrize("ty", RAGGED)
@pytest.mark.parametrize("k", [128, 896, 1152, 4224])
def test_rows_that_end_inside_a_unit_keep_fp32_precision(ctx, ty, k):
    """No further from float64 (2-norm over M x N results) than the plain kernels' fp32 sums, from which
    these rows were taken over; a tenth is left for the spread of the 6000 results' errors."""
    m, n = 2000, 3
    w = ctx.upload(synth.random_blocks(ty, m * k // block_elems(ty), np.random.default_rng(k)))
    t = GGUFTensor("w", (k, m), ty)
    W = torch.empty(m * k, device="cuda")
    CudaEnc(ctx).dequantRow(w, W, m * k, ty)
    X = torch.randn(n, k, device="cuda", generator=torch.Generator("cuda").manual_seed(k))
    exact = X.double() @ W.view(m, k).double().T
    err = []
    for flag in (0, 1):
        out = torch.empty(n, m, device="cuda")
        ctx.set_flags(flag)
        try:
            CudaEnc(ctx).gemm(t, X, out, w, n)
        finally:
            ctx.set_flags(0)
        err.append(float((out.double() - exact).norm() / exact.norm()))
    assert err[0] <= 1.1 * err[1], err


@pytest.mark.parametrize("ty", RAGGED)
def test_rows_that_end_inside_a_unit_at_the_ends_of_the_range(ctx, ty):
    """Activations near the smallest and the largest floats, subnormal ones, infinities and NaNs: as fp32 arithmetic
    has them.  Results below 2^-126 are held to steps of 2^-149 in any order of sums."""
    k, m = 1152, 64
    w = ctx.upload(synth.random_blocks(ty, m * k // block_elems(ty), np.random.default_rng(9)))
    t = GGUFTensor("w", (k, m), ty)
    W = torch.empty(m * k, device="cuda")
    CudaEnc(ctx).dequantRow(w, W, m * k, ty)
    W = W.view(m, k).double()
    base = torch.randn(k, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    out = torch.empty(m, device="cuda")
    for scale in (2.0 ** 60, 1e-20, 1e-31, 1e-36, 1e-40):
        x = base * scale
        CudaEnc(ctx).gemm(t, x, out, w, 1)
        exact = W @ x.double()
        assert (out.double() - exact).abs().max() <= RAGGED_TOL * exact.abs().max() + k * 2.0 ** -149, scale
    for value in (float("inf"), -float("inf"), float("nan")):
        x = base.clone()
        x[300] = value
        CudaEnc(ctx).gemm(t, x, out, w, 1)
        exact = (W @ x.double()).float()
        assert torch.equal(out.isnan(), exact.isnan()) and torch.equal(out.isinf(), exact.isinf())
        assert torch.equal(out[out.isinf()], exact[exact.isinf()])
