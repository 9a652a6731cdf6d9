"""The workloads this library's speed is judged by: whole calls through the
public entry points (fz::Pipeline, the batched launch, the per-chunk coder
selector) on seeded synthetic fields of the repository's benchmark shapes.

A case is a dict of plain values:
  op    "lbr"    LorenzoQuant -> Bitshuffle -> RZE through fz::Pipeline
        "rle"    LorenzoQuant -> RLE through fz::Pipeline
        "huff"   LorenzoQuant (radius 512) -> Huffman (1024 bins) through fz::Pipeline
        "pfpl"   Quantizer -> Difference -> Bitshuffle -> RZE through fz::Pipeline
        "batch"  many fields of mixed rank in one graph-captured batched launch
        "select" quantization codes through the learned per-chunk coder selector
  way   "enc" (compress), "dec" (decompress) or "both" (compress, then
        decompress what came out)
  x, y, z, eb, mode ("ABS", "REL", "NOA"), spikes (share of cells set to +-1e3)
        the field and its error bound; for "batch": count, low_mb, high_mb.
"""
import math
import random

import numpy as np
import torch

from fzgpumodules_b200 import fields as F
from fzgpumodules_b200 import kernels as K
from fzgpumodules_b200 import pipeline as P
from fzgpumodules_b200 import selector as S

MODES = {"ABS": P.ABS, "REL": P.REL, "NOA": P.NOA}


def _case(op, way, x, y=1, z=1, eb=1e-3, mode="REL", spikes=0.0):
    return {"op": op, "way": way, "x": x, "y": y, "z": z, "eb": eb, "mode": mode, "spikes": spikes}


def listed():
    return [
        # a small block of a simulation saved between steps: the call's latency counts
        dict(_case("lbr", "both", 64, 64, 64, 1e-3, "REL", 1e-3), name="block64"),
        # the Quick Start chain on a climate-sized 2-D field
        dict(_case("rle", "both", 3600, 1800, 1, 1e-4, "ABS"), name="plane-rle"),
        # the command line tool's documented configuration on the same field
        dict(_case("lbr", "both", 3600, 1800, 1, 1e-3, "REL"), name="plane-rze"),
        # the flagship chain on a whole simulation snapshot, each direction
        dict(_case("lbr", "enc", 512, 512, 512, 1e-3, "REL", 1e-3), name="cube512-enc"),
        dict(_case("lbr", "dec", 512, 512, 512, 1e-3, "REL", 1e-3), name="cube512-dec"),
        # a snapshot whose sides are no powers of two, an absolute bound and outliers
        dict(_case("lbr", "enc", 500, 500, 100, 1e-2, "ABS", 1e-3), name="ragged-enc"),
        dict(_case("lbr", "dec", 500, 500, 100, 1e-2, "ABS", 1e-3), name="ragged-dec"),
        # entropy-coded archive of a large image-like field, each direction
        dict(_case("huff", "enc", 8192, 8192, 1, 1e-3, "ABS"), name="huff8192-enc"),
        dict(_case("huff", "dec", 8192, 8192, 1, 1e-3, "ABS"), name="huff8192-dec"),
        # the point-wise relative preset, there and back
        dict(_case("pfpl", "both", 512, 512, 256, 1e-3, "REL", 1e-3), name="pfpl"),
        # a checkpoint of many arrays of uneven size in one launch
        {"op": "batch", "count": 20, "low_mb": 1, "high_mb": 256, "name": "batch20"},
        # mixed data coded by the learned selector and read back
        dict(_case("select", "both", 256, 256, 256, 1e-3, "REL"), name="select"),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng: random.Random):
    """Another field size, rank, bound and direction of the same chains."""
    op = rng.choice(["lbr", "lbr", "lbr", "lbr", "rle", "huff", "huff", "pfpl", "batch", "select"])
    way = rng.choice(["enc", "dec", "both"])
    mode, eb = rng.choice([("REL", 1e-2), ("REL", 1e-3), ("REL", 1e-4), ("ABS", 1e-2), ("ABS", 1e-3), ("NOA", 1e-3)])
    if op == "batch":
        low = rng.choice([1, 2, 4])
        return {"op": op, "count": rng.randint(4, 20), "low_mb": low, "high_mb": _log_int(rng, 2 * low, 256)}
    if op == "select":
        return _case(op, "both", rng.choice([96, 128, 200, 256]), rng.randint(40, 256), rng.randint(40, 256), eb, "REL")
    if op == "rle":
        x = _log_int(rng, 300, 6000)
        return _case(op, way, x, _log_int(rng, 300, 6000), 1, rng.choice([1e-4, 1e-3]), rng.choice(["ABS", "REL"]))
    if op == "huff":
        x = rng.choice([2048, 4096, 8192, rng.randint(1500, 8192)])
        return _case(op, way, x, rng.randint(1500, 8192), 1, 1e-3, "ABS")
    n = _log_int(rng, 1 << 18, 1 << 26)
    spikes = rng.choice([0.0, 1e-3])
    if op == "pfpl":
        return _case(op, way, n, 1, 1, rng.choice([1e-2, 1e-3]), "REL", spikes)
    rank = rng.choice([1, 2, 2, 3, 3, 3])
    if rank == 1:
        return _case(op, way, n, 1, 1, eb, mode, spikes)
    if rank == 2:
        x = rng.choice([256, 1024, 4096, rng.randint(200, 9000)])
        return _case(op, way, x, max(n // x, 2), 1, eb, mode, spikes)
    x = rng.choice([64, 128, 256, 512, rng.randint(40, 640), rng.randint(40, 640)])
    y = rng.choice([64, 128, 256, rng.randint(40, 640), rng.randint(40, 640)])
    return _case(op, way, x, y, max(n // (x * y), 2), eb, mode, spikes)


def _up(v):
    """The next size whose only prime factors are 2 and 3."""
    best = 1
    while best < v:
        best *= 2
    t = 3
    while t < best:
        p = t
        while p < v:
            p *= 2
        best, t = min(best, p), t * 3
    return best


def _smooth(dims, seed, spikes, dev):
    """A Gaussian random field k^-3 of x, y, z extents `dims`, cut from one of
    FFT-friendly extents, with spikes."""
    shape = [int(d) for d in reversed(dims) if d > 1] or [int(dims[0])]
    big = F.grf([_up(s) for s in shape], seed=seed, device=dev)
    v = big[tuple(slice(0, s) for s in shape)].contiguous().reshape(-1)
    if spikes > 0:
        g = torch.Generator(device=dev).manual_seed(seed + 77)
        m = max(1, int(v.numel() * spikes))
        at = torch.randint(0, v.numel(), (m,), generator=g, device=dev).unique()
        sign = torch.where(torch.rand(at.numel(), generator=g, device=dev) < 0.5, -1e3, 1e3)
        v[at] = sign.to(torch.float32)
    return v


def _field(case, seed, dev):
    d = (case["x"], case["y"], case["z"])
    if case["op"] == "rle" or (case["op"] == "lbr" and d == (3600, 1800, 1)):
        return F.sinusoids2d(d[1], d[0], seed=seed, device=dev).reshape(-1)
    if case["op"] == "huff":
        side = max(d[0], d[1])
        return F.fractal2d(side, seed=seed, device=dev)[: d[1], : d[0]].contiguous().reshape(-1)
    return _smooth(d, seed, case["spikes"], dev)


def _pipeline(case, n):
    pl = P.Pipeline(4 * n, P.PREALLOCATE)
    pl.setDims(case["x"], case["y"], case["z"])
    op, eb, mode = case["op"], case["eb"], MODES[case["mode"]]
    if op == "lbr":
        a = pl.addStage(P.LorenzoQuantStage(eb, 32768, 0.1, mode, True))
        b = pl.addStage(P.BitshuffleStage(16384, 2))
        c = pl.addStage(P.RZEStage(16384, 4))
        pl.connect(b, a, "codes")
        pl.connect(c, b)
    elif op == "rle":
        a = pl.addStage(P.LorenzoQuantStage(eb, 32768, 0.2, mode, False))
        pl.connect(pl.addStage(P.RLEStage(2)), a, "codes")
    elif op == "huff":
        a = pl.addStage(P.LorenzoQuantStage(eb, 512, 0.2, mode, True))
        pl.connect(pl.addStage(P.HuffmanStage(1024)), a, "codes")
    else:
        a = pl.addStage(P.QuantizerStage(eb, mode, 32768, 0.1, code_bytes=4, zigzag_codes=True))
        b = pl.addStage(P.DifferenceStage(P.INT32, P.UINT32, 16384))
        c = pl.addStage(P.BitshuffleStage(16384, 2))
        d = pl.addStage(P.RZEStage(16384, 4))
        pl.connect(b, a, "codes")
        pl.connect(c, b)
        pl.connect(d, c)
    pl.finalize()
    return pl


def _batch_dims(case):
    """Sizes spread over the logarithm of the case's range, ranks, extents and
    bounds mixed, the same for every seed."""
    k = case["count"]
    rng = np.random.default_rng(k)
    out = []
    for i in range(k):
        t = (i + 0.5) / k
        mb = case["low_mb"] * (case["high_mb"] / case["low_mb"]) ** t
        n = int(mb * (1 << 18))
        rank = 1 + (i * 7 + 2) % 3
        if rank == 1:
            out.append((n, 1, 1))
        elif rank == 2:
            nx = int(rng.choice([256, 512, 1000, 1024, 2048, 3000]))
            out.append((nx, max(n // nx, 2), 1))
        else:
            nx, ny = int(rng.choice([64, 128, 200, 256, 512])), int(rng.choice([64, 100, 128, 256]))
            out.append((nx, ny, max(n // (nx * ny), 2)))
    return out, [float(v) for v in rng.choice([1e-2, 1e-3, 1e-4], k)]


def _select_params(sel, codes, eb):
    """Weights for the selector: its seeded hidden layers with the output layer
    fitted by ridge regression in 64 bits to the log sizes of the codes' own
    chunks (the same for the same codes, which stochastic training is not)."""
    x = S.features(codes).double()
    t = S.targets_from_sizes(S.trial_sizes(codes)).double()
    p = sel.params.double()
    w1, b1 = p[:1024].view(16, 64), p[1024:1088]
    w2, b2 = p[1088:5184].view(64, 64), p[5184:5248]
    h = torch.relu(torch.relu(x @ w1 + b1) @ w2 + b2)
    h = torch.cat([h, torch.ones_like(h[:, :1])], 1)
    w = torch.linalg.solve(h.T @ h + 1e-6 * h.shape[0] * torch.eye(65, device=h.device, dtype=h.dtype), h.T @ t)
    sel.params[5248:] = torch.cat([w[:64].reshape(-1), w[64]]).float()


# bytes per value that a program sets aside for a stream of each chain
_ROOM = {"lbr": 3, "rle": 8, "huff": 4, "pfpl": 6}


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    if case["op"] == "batch":
        dims, ebs = _batch_dims(case)
        fields = [dict(x=_smooth(d, seed * 1000 + i, 1e-3, dev), dims=d, eb=e, mode=K.REL, radius=32768, zigzag=True,
                       outlier_capacity=0.1) for i, (d, e) in enumerate(zip(dims, ebs))]
        b = K.Batch(fields)
        for o in b.outputs:  # what lies past a stream's end is not part of it
            for t in (o["rze"], o["err"], o["idx"]):
                t.zero_()
        s = torch.cuda.Stream(device=dev)
        s.wait_stream(torch.cuda.current_stream(dev))
        b.launch(s)
        s.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            b.launch(s)
        return {"case": case, "batch": b, "graph": g}
    n = case["x"] * case["y"] * case["z"]
    if case["op"] == "select":
        dims = (case["x"], case["y"], case["z"])
        codes = []
        for i, kind in enumerate(("smooth", "piecewise", "noise", "sparse")):
            v = _smooth(dims, seed * 1000, 0.0, dev) if kind == "smooth" else F.mixed_field(kind, dims[::-1], seed * 1000 + i, device=dev)
            codes.append(K.lq_forward(v, dims, case["eb"], K.REL, 32768, True, 0.2)["codes"].view(torch.int16))
        codes = torch.cat(codes).view(torch.uint16)
        sel = S.CoderSelector(seed=0, device=dev)
        _select_params(sel, codes, case["eb"])
        keep = torch.zeros(codes.numel() * 2 + (1 << 16), dtype=torch.uint8, device=dev)
        return {"case": case, "codes": codes, "sel": sel, "keep": keep}
    x = _field(case, seed, dev)
    pl = _pipeline(case, n)
    st = {"case": case, "x": x, "n": n, "pl": pl}
    if case["way"] == "dec":
        st["comp"] = pl.compress(x).clone()
    else:
        st["keep"] = torch.zeros(_ROOM[case["op"]] * n + (1 << 20), dtype=torch.uint8, device=dev)
    return st


class _Held(list):
    """Outputs that are views of a pipeline's own memory, and the pipeline."""

    def __init__(self, outputs, pipeline):
        super().__init__(outputs)
        self.pipeline = pipeline


def run(state):
    case = state["case"]
    if case["op"] == "batch":
        state["graph"].replay()
        outs = state["batch"].outputs
        sizes = torch.cat([o["rze_size"] for o in outs] + [o["count"].to(torch.int64) for o in outs])
        return [sizes] + [[o["rze"], o["err"], o["idx"]] for o in outs]
    keep = state.get("keep")
    if case["op"] == "select":
        blob, tags = S.encode(state["codes"], S.LEARNED, state["sel"])
        keep[: blob.numel()].copy_(blob)
        return [keep, blob.numel(), tags, S.decode(blob, state["codes"].numel()).view(torch.int16)]
    pl, n = state["pl"], state["n"]
    if case["way"] == "dec":
        return _Held([pl.decompress(state["comp"])[:n]], pl)
    comp = pl.compress(state["x"])
    nb = comp.numel()
    keep[:nb].copy_(comp)  # the pipeline's view is good until its next call: the program keeps the bytes
    if case["way"] == "enc":
        return [keep, nb]
    return _Held([keep, nb, pl.decompress(keep[:nb])[:n]], pl)


# compressed bytes per value, about what these fields give: the work counts the
# field or codes once and the compressed stream once
_STREAM = {"lbr": 0.5, "rle": 5.8, "huff": 0.3, "pfpl": 3.2}


def work(case):
    if case["op"] == "batch":
        return {"bytes": 4.15 * sum(x * y * z for x, y, z in _batch_dims(case)[0]), "flops": 0}
    n = case["x"] * case["y"] * case["z"]
    if case["op"] == "select":
        return {"bytes": 2 * 4 * n * (2 + 2 / 2.3), "flops": 0}
    return {"bytes": (2 if case["way"] == "both" else 1) * n * (4 + _STREAM[case["op"]]), "flops": 0}


def tolerance(case):
    """Streams, codes and reconstructions are defined bit for bit."""
    return "exact"


def exact(case, seed):
    """The reconstruction each chain defines, in 64 bits; streams have none."""
    if case["op"] in ("batch", "select") or case["way"] == "enc":
        return None
    x = _field(case, seed, torch.device("cuda", torch.cuda.current_device()))
    if case["op"] == "pfpl":
        log2eb = float(np.float32(2) * np.log2(np.float32(1) + np.float32(case["eb"])))  # the preset's 32-bit bin width
        v = x.double()
        y = torch.sign(v) * torch.exp2(torch.round(torch.log2(v.abs()) / log2eb) * log2eb)
        y = torch.where(v == 0, v, y)
    else:
        eb = np.float32(case["eb"])
        lo, hi = (np.float32(float(t)) for t in (x.min(), x.max()))
        base = {"ABS": np.float32(1), "REL": max(abs(lo), abs(hi)), "NOA": hi - lo}[case["mode"]]
        a = eb * base
        t = (x * float(np.float32(1) / (np.float32(2) * a))).double()  # the quantizer's 32-bit product, exact from here
        q = torch.sign(t) * torch.floor(t.abs() + 0.5)
        y = q * float(np.float32(2) * a)
    return [y] if case["way"] == "dec" else [None, None, y]
