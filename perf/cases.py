"""The work that programs give this framework, as cases that can be timed.

Six kinds of pass cover the entry points of an inference engine built on the library:

  host     the host-buffer operator on numpy arrays (the CPU engine's matvec / matmul)
  block    token ids -> embedding rows -> FFN blocks (residual add + RMS norm, gate || up,
           SiLU gating, down), all in fp32 as the operators hand them on
  linears  the linear projections of a trunk's layers on activations kept in 16 bits or
           fp32: q || k || v, o, gate || up, down
  matmul   one FFN pair (hidden -> inner, inner -> hidden) over a prompt chunk
  logits   final norm, output projection over the vocabulary, arg-max per row
  ragged   independent linears of odd heights and row lengths

Sizes are those of this repository's benchmark workloads and tests, or generic ones between
them.  Weights are blocks quantized from N(0, 0.02) (ternary: P = 1/4, 1/2, 1/4), drawn from
a pool by the seed; every layer owns its weights, so a decode pass reads them from HBM.
"""
import math

import numpy as np
import torch

from chatokf_b200 import synth
from chatokf_b200.enc import QB, Context, CudaEnc, GGUFTensor
from chatokf_b200.gguf_types import GGUFType, block_elems, row_byte_count

DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
VOCAB = 151936
EPS = 1e-6


def listed():
    return [
        # The smallest call: one 2048 x 2048 Q8_0 matvec from host memory to host memory, where
        # copies, launches and the wait for the result are all there is.
        dict(name="host_q8_0", kind="host", type="Q8_0", k=2048, m=2048, n=1),
        # Decode, one token: four FFN blocks of the 2560 / 9728 shape behind the embedding.
        dict(name="block_q4_k_decode", kind="block", type="Q4_K", hidden=2560, inner=9728, layers=4, n=1),
        # Decode, one token, through two layers of a 27B-shaped two-bit trunk.
        dict(name="trunk_iq2_xxs_decode", kind="linears", type="IQ2_XXS", hidden=5120, kv=1024, inner=17408, layers=2, n=1,
             x="f16"),
        # The same trunk verifying four drafted tokens at once.
        dict(name="trunk_iq2_xxs_verify4", kind="linears", type="IQ2_XXS", hidden=5120, kv=1024, inner=17408, layers=2, n=4,
             x="f16"),
        # The widest verify batch.
        dict(name="block_q4_k_verify8", kind="block", type="Q4_K", hidden=2560, inner=9728, layers=4, n=8),
        # Decode through a small ternary model: matrices of 1 to 3 MB, where launches count.
        dict(name="trunk_q2_0_decode", kind="linears", type="Q2_0", hidden=2048, kv=1024, inner=6144, layers=8, n=1, x="f16"),
        # Odd sizes: rows that are no multiple of 256 weights, heights that are no multiple of a tile.
        dict(name="ragged_q4_0", kind="ragged", type="Q4_0", k=1056, m=5003, count=6, n=3, x="f32"),
        # Prompt processing, a chunk of 512 tokens, bf16 activations.
        dict(name="matmul_q4_k_512", kind="matmul", type="Q4_K", hidden=5120, inner=17408, n=512, x="bf16", out="f32"),
        # The ternary model's prompt chunk, fp16 activations.
        dict(name="matmul_q2_0_512", kind="matmul", type="Q2_0", hidden=2048, inner=6144, n=512, x="f16", out="f32"),
        # The largest: a long prompt at once, results kept in bf16.
        dict(name="matmul_q4_k_4096", kind="matmul", type="Q4_K", hidden=5120, inner=17408, n=4096, x="bf16", out="bf16"),
        # A short prompt of odd length through the fp32 operators, five-bit weights.
        dict(name="block_q5_k_prompt77", kind="block", type="Q5_K", hidden=2560, inner=9728, layers=2, n=77),
        # The end of every decode step: logits over the vocabulary and the greedy token.
        dict(name="logits_q6_k", kind="logits", type="Q6_K", hidden=2560, vocab=VOCAB, n=1),
    ]


TYPES = ["Q8_0", "Q4_K", "Q4_K", "IQ2_XXS", "Q2_0", "Q4_0", "Q5_K", "Q6_K", "IQ4_NL"]
MOST_BYTES = 1 << 28  # of weights in a drawn case
MOST_FLOPS = 2 * 2 * 4096 * 5120 * 17408


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _row(rng, ty, lo, hi):
    """A row length: any whole number of blocks, most often a multiple of 256."""
    step = block_elems(GGUFType[ty]) if rng.random() < 0.3 else 256
    return max(step, round(_log(rng, lo, hi) / step) * step)


def _tokens(rng):
    """One token in decode, a verify batch, or a prompt."""
    p = rng.random()
    return 1 if p < 0.4 else rng.randint(2, 8) if p < 0.65 else round(_log(rng, 9, 2048))


def draw(rng):
    while True:
        kind = rng.choice(["block", "block", "linears", "linears", "matmul", "matmul", "logits", "ragged", "host"])
        ty = rng.choice(TYPES)
        c = dict(kind=kind, type=ty)
        if kind == "host":
            n = 1 if rng.random() < 0.5 else round(_log(rng, 2, 256))
            c.update(k=_row(rng, ty, 512, 8192), m=round(_log(rng, 256, 16384)), n=n)
        elif kind == "block":
            c.update(hidden=_row(rng, ty, 512, 6144), inner=_row(rng, ty, 1024, 18432), layers=rng.randint(1, 6), n=_tokens(rng))
        elif kind == "linears":
            n = 1 if rng.random() < 0.5 else rng.randint(2, 8)
            hidden = _row(rng, ty, 512, 6144)
            c.update(hidden=hidden, kv=max(64, hidden // rng.choice([2, 4, 5, 8]) // 64 * 64), inner=_row(rng, ty, 1024, 18432),
                     layers=rng.randint(1, 8), n=n, x=rng.choice(["f16", "bf16", "f32"]))
        elif kind == "matmul":
            c.update(hidden=_row(rng, ty, 512, 8192), inner=_row(rng, ty, 1024, 20480), n=round(_log(rng, 9, 4096)),
                     x=rng.choice(["bf16", "f16", "f32"]), out=rng.choice(["f32", "bf16"]))
        elif kind == "logits":
            c.update(hidden=_row(rng, ty, 512, 6144), vocab=round(_log(rng, 16384, 262144)), n=1 if rng.random() < 0.6 else rng.randint(2, 8))
        else:
            c.update(k=_row(rng, ty, 256, 8192), m=round(_log(rng, 100, 20000)), count=rng.randint(1, 6), n=_tokens(rng),
                     x=rng.choice(["f16", "bf16", "f32"]))
        if sum(_tensor_bytes(t) for t in _tensors(c)) <= MOST_BYTES and work(c)["flops"] <= MOST_FLOPS:
            return c


# ---- weights -------------------------------------------------------------------------------

def _tensors(c):
    """The matrices of a case as (K, M, type), in the order they lie in the buffer."""
    ty, kind = GGUFType[c["type"]], c["kind"]
    if kind == "host":
        return [(c["k"], c["m"], ty)]
    if kind == "block":
        h, f = c["hidden"], c["inner"]
        return [(h, 4096, ty)] + [(h, f, ty), (h, f, ty), (f, h, ty)] * c["layers"]
    if kind == "linears":
        h, f, kv = c["hidden"], c["inner"], c["kv"]
        return [(h, h, ty), (h, kv, ty), (h, kv, ty), (h, h, ty), (h, f, ty), (h, f, ty), (f, h, ty)] * c["layers"]
    if kind == "matmul":
        return [(c["hidden"], c["inner"], ty), (c["inner"], c["hidden"], ty)]
    if kind == "logits":
        return [(c["hidden"], c["vocab"], ty)]
    return [(c["k"], c["m"] + 7 * i, ty) for i in range(c["count"])]


def _tensor_bytes(t):
    k, m, ty = t
    return row_byte_count(ty, k) * m


_pools = {}


def _pool(ty):
    """Blocks to draw weights from, quantized once."""
    if ty not in _pools:
        rng = np.random.default_rng(int(ty))
        count = 1 << 13
        if ty == GGUFType.Q2_0:
            blocks = synth.ternary_q2_0(rng, count * block_elems(ty))
        else:
            blocks = synth.quantize(ty, rng.normal(0.0, 0.02, size=count * block_elems(ty)).astype(np.float32))
        _pools[ty] = torch.from_numpy(blocks.reshape(count, -1)).cuda()
    return _pools[ty]


def _weights(ctx, tensors, gen):
    """One device buffer with the tensors at multiples of 32 bytes, as in a GGUF data region."""
    offsets, at = [], 0
    for t in tensors:
        offsets.append(at)
        at += (_tensor_bytes(t) + 31) // 32 * 32
    buf = torch.zeros(at + 256, dtype=torch.uint8, device="cuda")
    for t, o in zip(tensors, offsets):
        pool = _pool(t[2])
        blocks = _tensor_bytes(t) // pool.shape[1]
        pick = torch.randint(0, pool.shape[0], (blocks,), device="cuda", generator=gen)
        torch.index_select(pool, 0, pick, out=buf[o:o + _tensor_bytes(t)].view(blocks, pool.shape[1]))
    views = [GGUFTensor("w%d" % i, (k, m), ty, o) for i, ((k, m, ty), o) in enumerate(zip(tensors, offsets))]
    return ctx.wrap(buf, at), views


_ctx = None


def _context():
    """A program keeps one context."""
    global _ctx
    if _ctx is None:
        _ctx = Context(torch.cuda.current_device())
    return _ctx


# ---- passes --------------------------------------------------------------------------------

def prepare(case, seed):
    c = dict(case)
    kind, n = c["kind"], c["n"]
    ctx = _context()
    gen = torch.Generator(device="cuda").manual_seed(int(seed))

    def normal(*shape, dtype=torch.float32):
        return torch.randn(*shape, device="cuda", generator=gen).to(dtype)

    def empty(*shape, dtype=torch.float32):
        return torch.zeros(*shape, dtype=dtype, device="cuda")

    off, w = _weights(ctx, _tensors(c), gen)
    s = dict(case=c, off=off, w=w, enc=CudaEnc(ctx))
    if kind == "host":
        rng = np.random.default_rng(int(seed))
        s.update(qb=QB(ctx), x=rng.normal(size=(n, c["k"])).astype(np.float32), out=np.zeros((n, c["m"]), np.float32))
    elif kind == "block":
        h, f, layers = c["hidden"], c["inner"], c["layers"]
        s.update(ids=torch.randint(0, 4096, (n,), device="cuda", generator=gen, dtype=torch.int32),
                 norms=[1.0 + 0.1 * normal(h) for _ in range(layers + 1)], x=empty(n, h), y=empty(n, h), gate=empty(n, f),
                 up=empty(n, f), down=empty(n, h))
    elif kind == "linears":
        h, f, kv, dt = c["hidden"], c["inner"], c["kv"], DTYPES[c["x"]]
        s.update(xs=[[normal(n, h, dtype=dt), normal(n, h, dtype=dt), normal(n, h, dtype=dt), normal(n, f, dtype=dt)]
                     for _ in range(c["layers"])],
                 outs=[[empty(n, m) for m in (h, kv, kv, h, f, f, h)] for _ in range(c["layers"])])
    elif kind == "matmul":
        h, f, dt, odt = c["hidden"], c["inner"], DTYPES[c["x"]], DTYPES[c["out"]]
        s.update(xh=normal(n, h, dtype=dt), xf=normal(n, f, dtype=dt), up=empty(n, f, dtype=odt), down=empty(n, h, dtype=odt))
    elif kind == "logits":
        s.update(x=normal(n, c["hidden"]), norm=1.0 + 0.1 * normal(c["hidden"]), y=empty(n, c["hidden"]),
                 logits=empty(n, c["vocab"]), ids=torch.zeros(n, dtype=torch.int32, device="cuda"))
    else:
        s.update(xs=[normal(n, c["k"], dtype=DTYPES[c["x"]]) for _ in w], outs=[empty(n, t.M) for t in w])
    return s


def run(s):
    c, w, off, enc = s["case"], s["w"], s["off"], s["enc"]
    kind, n = c["kind"], c["n"]
    if kind == "host":
        return s["qb"].matmul(w[0], off, s["x"], n, out=s["out"])
    if kind == "block":
        h, f = c["hidden"], c["inner"]
        x, y, gate, up, down = s["x"], s["y"], s["gate"], s["up"], s["down"]
        enc.embedBatch(s["ids"], off, x, h, n, w[0].type, 4096, w[0].offset)
        residual = None
        for i in range(c["layers"]):
            enc.addRmsnormBatch(x, residual, s["norms"][i], y, h, n, EPS)
            with enc.parallel():
                enc.gemm(w[3 * i + 1], y, gate, off, n)
                enc.gemm(w[3 * i + 2], y, up, off, n)
            enc.siluMul(gate, up, n * f)
            enc.gemm(w[3 * i + 3], gate, down, off, n)
            residual = down
        enc.addRmsnormBatch(x, residual, s["norms"][-1], y, h, n, EPS)
        return {"x": x, "y": y, "gate": gate, "up": up, "down": down}
    if kind == "linears":
        for i in range(c["layers"]):
            xs, outs, t = s["xs"][i], s["outs"][i], w[7 * i:7 * i + 7]
            with enc.parallel():
                for j in range(3):
                    enc.gemm(t[j], xs[0], outs[j], off, n)
            enc.gemm(t[3], xs[1], outs[3], off, n)
            with enc.parallel():
                enc.gemm(t[4], xs[2], outs[4], off, n)
                enc.gemm(t[5], xs[2], outs[5], off, n)
            enc.gemm(t[6], xs[3], outs[6], off, n)
        return s["outs"]
    if kind == "matmul":
        enc.gemm(w[0], s["xh"], s["up"], off, n)
        enc.gemm(w[1], s["xf"], s["down"], off, n)
        return {"up": s["up"], "down": s["down"]}
    if kind == "logits":
        enc.addRmsnormBatch(s["x"], None, s["norm"], s["y"], c["hidden"], n, EPS)
        enc.gemm(w[0], s["y"], s["logits"], off, n)
        enc.argmaxRows(s["logits"], s["ids"], c["vocab"], n)
        return {"logits": s["logits"], "ids": s["ids"]}
    for t, x, out in zip(w, s["xs"], s["outs"]):
        enc.gemm(t, x, out, off, n)
    return s["outs"]


def work(case):
    c = case
    n, tensors, kind = c["n"], _tensors(c), c["kind"]
    xs, osz = {"f32": 4, "f16": 2, "bf16": 2}[c.get("x", "f32")], 2 if c.get("out") == "bf16" else 4
    mats = tensors[1:] if kind == "block" else tensors
    weights = sum(_tensor_bytes(t) for t in mats)
    flops = sum(2 * n * k * m for k, m, _ in mats)
    if kind == "host":
        moved = n * (c["k"] + c["m"]) * 4
    elif kind == "block":
        # embedding rows in, the last residual, norm, gate, up and down out, the norms' weights
        moved = n * row_byte_count(tensors[0][2], c["hidden"]) + (c["layers"] + 1) * c["hidden"] * 4
        moved += n * (3 * c["hidden"] + 2 * c["inner"]) * 4
    elif kind == "linears":
        moved = c["layers"] * n * ((3 * c["hidden"] + c["inner"]) * xs + sum(m for _, m, _ in tensors[:7]) * 4)
    elif kind == "matmul":
        moved = n * (c["hidden"] + c["inner"]) * (xs + osz)
    elif kind == "logits":
        moved = n * (2 * c["hidden"] * 4 + c["vocab"] * 4 + 4) + c["hidden"] * 4
    else:
        moved = sum(n * (k * xs + m * 4) for k, m, _ in tensors)
    return {"bytes": weights + moved, "flops": flops}


def tolerance(case):
    """Up to eight tokens activations carry 16 bits (a step of 2^-15 of the largest of 256) and sums
    are exact; beyond, both operands are rounded to fp16 (fp16 activations) or bf16 once."""
    n, kind = case["n"], case["kind"]
    if n <= 8 and case.get("out") != "bf16":
        return {"rel": 2e-4 if kind == "block" else 1e-4}  # a block's errors pass through its later linears
    if kind == "block":
        return {"rel": 1e-2}
    if case.get("out") == "bf16":
        return {"rel": 5e-3}
    return {"rel": 5e-4 if case.get("x") == "f16" else 4e-3}
