"""The framework's work as its users have it done, at sizes from the smallest call to the largest.

A case is a dict: its "kind" names the entry point, the rest are sizes and options.

  matvec   Q8Matrix.matvec: one int8 matrix in the Q8 layout, 1..64 int8 vectors, optionally with per-row scales
  stack    Q8Stack.run: the seven matrices of a transformer layer, each with its own input, in one launch
  chain    Q8Chain.run: matrices applied in turn, requantised to int8 between them
  linear   q8_linear under autograd: the float form, forward and backward
  awr      AwrMatrix.matvec_requant (one vector) or .matvec: the reference's ans-warp-rows files
  wpr      WprMatrix.matvec, then requant_absmax: the reference's matvansWarpPerRow files
  aws      AwsMatrix.matvec_requant (one vector) or .matvec: the reference's ans-warp-stripes files

Weights are rounded Gaussians (or Laplace with rare outliers), as quantised layers have them.
"""
import math

import numpy as np
import torch

from matvans_b200 import autograd, ops

DEV = "cuda"


def listed():
    return [
        # the smallest matrix a program keeps compressed; one vector, where latency and launches count
        dict(name="small_1024", kind="matvec", rows=1024, cols=1024, batch=1, local=True, dist="gauss", sigma=4.0,
             scaled=False),
        # the largest single matrix (a 70B model's up projection), low entropy, one vector
        dict(name="large_28672x8192", kind="matvec", rows=28672, cols=8192, batch=1, local=True, dist="laplace",
             sigma=2.0, scaled=False),
        # a prompt of 64 tokens through one 7B projection, scaled outputs
        dict(name="prompt_b64", kind="matvec", rows=11008, cols=4096, batch=64, local=True, dist="gauss", sigma=4.0,
             scaled=True),
        # a matrix whose sides fit no tile, one table for all rows, two sequences decoding
        dict(name="ragged_4090x4100_b2", kind="matvec", rows=4090, cols=4100, batch=2, local=False, dist="gauss",
             sigma=2.0, scaled=False),
        # single-sequence decode: every matrix of a 7B layer in one launch
        dict(name="layer_b1", kind="stack", hidden=4096, ffn=11008, batch=1),
        # batched decode, 16 sequences
        dict(name="layer_b16", kind="stack", hidden=4096, ffn=11008, batch=16),
        # the reference's end-to-end program: matrices chained through the int8 requantisation
        dict(name="chain_b1", kind="chain", hidden=4096, ffn=11008, batch=1),
        # float form with its gradient: one token, and a small training batch
        dict(name="linear_b1", kind="linear", rows=4096, cols=11008, batch=1, local=True, sigma=4.0),
        dict(name="linear_b64", kind="linear", rows=11008, cols=4096, batch=64, local=True, sigma=4.0),
        # the reference's three stream layouts, one vector through the reference's own epilogue
        dict(name="awr_4096", kind="awr", rows=4096, cols=4096, batch=1, sigma=4.0),
        dict(name="wpr_4096", kind="wpr", rows=4096, cols=4096, batch=1, sigma=4.0),
        dict(name="aws_4096", kind="aws", rows=4096, cols=4096, batch=1, sigma=4.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the same kinds: sizes spread over their logarithm, odd ones among them, at most 64 M weights."""
    kind = rng.choice(["matvec", "matvec", "matvec", "stack", "stack", "chain", "linear", "linear", "awr", "wpr", "aws"])
    sigma = round(rng.uniform(1.0, 6.0), 2)
    local = rng.random() < 0.7
    if kind in ("stack", "chain"):
        hidden = 16 * _log(rng, 16, 176)
        return dict(kind=kind, hidden=hidden, ffn=16 * max(1, round(hidden * rng.uniform(2.0, 4.0) / 16)),
                    batch=_log(rng, 1, 16))
    cols = _log(rng, 256, 12000)
    rows = _log(rng, 64, min(16384, 64 * 2 ** 20 // cols))
    if kind == "matvec":
        if rng.random() < 0.8:
            cols = max(16, cols // 16 * 16)
        return dict(kind=kind, rows=rows, cols=cols, batch=_log(rng, 1, 64), local=local,
                    dist=rng.choice(["gauss", "gauss", "laplace"]), sigma=sigma, scaled=rng.random() < 0.4)
    if kind == "linear":
        return dict(kind=kind, rows=rows, cols=max(16, cols // 16 * 16), batch=_log(rng, 1, 64), local=local, sigma=sigma)
    batch = rng.choice([1, 1, 1, 2, 4, 16])
    if kind == "awr":
        return dict(kind=kind, rows=rows, cols=max(128, cols // 128 * 128), batch=batch, sigma=sigma)
    if kind == "wpr":
        return dict(kind=kind, rows=rows, cols=max(512, cols // 512 * 512), batch=batch, sigma=sigma)
    # a stripe is one sequential stream: rows set the parallelism, columns the length
    return dict(kind=kind, rows=max(32, rows // 32 * 32), cols=max(64, min(cols, 4096) // 4 * 4), batch=batch, sigma=sigma)


# ------------------------------------------------------------------ inputs, made from the seed alone

def _gen(seed, k=0):
    g = torch.Generator(device=DEV)
    g.manual_seed(1000003 * int(seed) + k)
    return g


def _weights(g, rows, cols, dist, sigma):
    if dist == "laplace":
        z = torch.empty((rows, cols), device=DEV).exponential_(generator=g)
        z -= torch.empty((rows, cols), device=DEV).exponential_(generator=g)
        z *= sigma
    else:
        z = torch.randn((rows, cols), device=DEV, generator=g) * sigma
    return z.round_().clamp_(-127, 127).to(torch.int8)


def _x8(g, batch, cols):
    return torch.randint(-127, 128, (batch, cols), dtype=torch.int8, device=DEV, generator=g)


def _row_scales(g, rows):
    return torch.rand(rows, device=DEV, generator=g) * 9e-3 + 1e-3


def _shapes(case):
    h, f = case["hidden"], case["ffn"]
    if case["kind"] == "chain":
        return [(h, h), (f, h), (h, f)]
    return [(h, h)] * 4 + [(f, h)] * 2 + [(h, f)]


def _layer_weights(case, seed, i, shape):
    """Matrix i of a layer: its own width, one in ten with heavy tails."""
    r = np.random.default_rng([int(seed), i])
    sigma, tails = float(r.uniform(2, 6)), r.random() < 0.1
    return _weights(_gen(seed, 10 + i), *shape, "laplace" if tails else "gauss", 3.0 if tails else sigma)


CHAIN_SCALE = 2e-3
AWR_SCALE = 2e-3


def _single(case, seed):
    g = _gen(seed)
    W = _weights(g, case["rows"], case["cols"], case.get("dist", "gauss"), case["sigma"])
    return g, W


def prepare(case, seed):
    kind, batch = case["kind"], case["batch"]
    st = {"kind": kind, "batch": batch}
    if kind in ("stack", "chain"):
        mats = [ops.Q8Matrix.encode(_layer_weights(case, seed, i, s).cpu().numpy(), device=DEV)
                for i, s in enumerate(_shapes(case))]
        g = _gen(seed)
        if kind == "stack":
            st["plan"] = ops.Q8Stack(mats, batch=batch, xs=[_x8(g, batch, M.cols) for M in mats], device=DEV)
        else:
            st["plan"] = ops.Q8Chain(mats, [CHAIN_SCALE] * len(mats), batch=batch, x0=_x8(g, batch, mats[0].cols),
                                     device=DEV)
        return st
    g, W = _single(case, seed)
    host = W.cpu().numpy()
    del W
    if kind == "linear":
        st["M"] = ops.Q8Matrix.encode(host, local=case["local"], device=DEV)
        st["scales"] = _row_scales(g, case["rows"])
        st["x"] = torch.randn((batch, case["cols"]), device=DEV, generator=g).to(torch.bfloat16).requires_grad_()
        st["gy"] = torch.randn((batch, case["rows"]), device=DEV, generator=g)
        return st
    if kind == "matvec":
        st["M"] = ops.Q8Matrix.encode(host, local=case["local"], device=DEV)
        st["scales"] = _row_scales(g, case["rows"]) if case["scaled"] else None
    else:
        st["M"] = {"awr": ops.AwrMatrix, "wpr": ops.WprMatrix, "aws": ops.AwsMatrix}[kind].encode(host, device=DEV)
    st["x"] = _x8(g, batch, case["cols"])
    return st


def run(state):
    kind = state["kind"]
    if kind == "matvec":
        return state["M"].matvec(state["x"], scales=state["scales"])
    if kind == "stack":
        return state["plan"].run()
    if kind == "chain":
        out8 = state["plan"].run()
        return [out8] + state["plan"].ys
    if kind == "linear":
        y = autograd.q8_linear(state["x"], state["M"], state["scales"])
        (dx,) = torch.autograd.grad(y, state["x"], state["gy"])
        return [y.detach(), dx]
    if kind == "wpr":
        y = state["M"].matvec(state["x"])
        return [y] + list(ops.requant_absmax(y))
    if state["batch"] == 1:
        return state["M"].matvec_requant(state["x"], AWR_SCALE)
    return state["M"].matvec(state["x"])


# ------------------------------------------------------------------ the same in 64 bits

def _mul(x, W):
    return (x.double() @ W.double().T).round().to(torch.int64)


def _requant(y, scale):
    """clamp(round half to even of the fp32 product): the reference's epilogue."""
    return (y.to(torch.float32) * torch.tensor(scale, dtype=torch.float32, device=DEV)).round().clamp(-128, 127).to(torch.int8)


def exact(case, seed):
    kind, batch = case["kind"], case["batch"]
    g = _gen(seed)
    if kind == "stack":
        shapes = _shapes(case)
        xs = [_x8(g, batch, c) for _, c in shapes]
        return [_mul(x, _layer_weights(case, seed, i, s)) for i, (x, s) in enumerate(zip(xs, shapes))]
    if kind == "chain":
        x, ys = _x8(g, batch, case["hidden"]), []
        for i, s in enumerate(_shapes(case)):
            ys.append(_mul(x, _layer_weights(case, seed, i, s)))
            x = _requant(ys[-1], CHAIN_SCALE)
        return [x] + ys
    g, W = _single(case, seed)
    if kind == "linear":
        s = _row_scales(g, case["rows"]).double()
        x = torch.randn((batch, case["cols"]), device=DEV, generator=g).to(torch.bfloat16).double()
        gy = torch.randn((batch, case["rows"]), device=DEV, generator=g).to(torch.bfloat16).double()
        W = W.double()
        return [(x @ W.T) * s, (gy * s) @ W]
    if kind == "matvec":
        s = _row_scales(g, case["rows"]).double() if case["scaled"] else None
        y = _mul(_x8(g, batch, case["cols"]), W)
        return y if s is None else (y, y.double() * s)
    y = _mul(_x8(g, batch, case["cols"]), W)
    if kind == "wpr":
        return [y, None, (y.abs().max().double() / 127).reshape(1)]
    return y if batch > 1 else _requant(y[0], AWR_SCALE)


# ------------------------------------------------------------------ what a pass cannot do without

def _bits(dist, sigma):
    """Entropy of one weight in bits."""
    if dist == "laplace":
        return max(1.0, math.log2(2 * math.e * sigma))
    return max(1.0, math.log2(sigma * math.sqrt(2 * math.pi * math.e)))


def work(case):
    """The entropy-coded weights read once, inputs read once, outputs written once; a multiply and an add per weight and vector."""
    kind, b = case["kind"], case["batch"]
    if kind in ("stack", "chain"):
        shapes = _shapes(case)
        n = sum(r * c for r, c in shapes)
        io = sum(c + 4 * r for r, c in shapes) if kind == "stack" else case["hidden"] * 2 + 4 * sum(r for r, _ in shapes)
        return {"bytes": n * _bits("gauss", 4.0) / 8 + b * io, "flops": 2.0 * n * b}
    r, c = case["rows"], case["cols"]
    coded = r * c * _bits(case.get("dist", "gauss"), case["sigma"]) / 8
    if kind == "linear":  # x bf16 in, y fp32 out; gy fp32 in, dx bf16 out
        return {"bytes": coded + 4 * r + b * (2 * c + 4 * r + 4 * r + 2 * c), "flops": 4.0 * r * c * b}
    out = 4 * r * (2 if case.get("scaled") else 1)
    if kind in ("awr", "aws") and b == 1:
        out = r
    if kind == "wpr":
        out = 5 * r
    return {"bytes": coded + b * (c + out), "flops": 2.0 * r * c * b}
