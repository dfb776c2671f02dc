"""The measured workloads of ncarray_gb300: what a user's program calls, over the sizes it calls it with.

``listed()`` names one case per family, ``draw(rng)`` gives another case of the same ranges. A case is a dict of plain
values; ``prepare`` makes the arrays (and the plan or handle that a program keeps) from a seed, ``run`` is one pass through
the public entry points, ``work`` what the pass cannot do without, and ``exact`` its floating outputs in 64 bits.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import ncarray_gb300 as nca
from ncarray_gb300.batch import Batch, BatchExpr
from ncarray_gb300.hist import hist2d
from ncarray_gb300.stencil import Stencil, Stencil3D, laplacian7, laplacian27

_T = {"float32": torch.float32, "float64": torch.float64, "bfloat16": torch.bfloat16, "uint16": torch.uint16,
      "int32": torch.int32, "int64": torch.int64, "uint64": torch.uint64}
_SIZE = {"float32": 4, "float64": 8, "bfloat16": 2, "uint16": 2, "int32": 4, "int64": 8}


def listed():
    return [
        # the smallest call: an expression over a small image, built and materialised on every call
        {"name": "expr_small", "kind": "expr", "dtype": "float32", "h": 33, "w": 127},
        # a float64 expression stored with its axis-0 sum and max, then the totals of both (the 128^3 configuration)
        {"name": "expr_reduce_f64", "kind": "expr_reduce", "dtype": "float64", "n0": 128, "n1": 128, "n2": 128},
        # transposed and broadcast views fused, stored and reduced, with an int32 expression (the (8, 256, 256, 64) configuration)
        {"name": "views_fused", "kind": "views", "q": 8, "b": 256, "r": 256, "p": 64},
        # a region of interest of detector frames: (raw - dark) * gain, rows that start anywhere
        {"name": "frames_roi", "kind": "frames", "raw": "uint16", "out": "float32", "n": 96, "h": 512, "w": 1024,
         "y0": 1, "y1": 510, "x0": 3, "x1": 1018},
        # ten Jacobi steps of the 7-point Laplacian on the 512^3 configuration
        {"name": "jacobi_7pt", "kind": "jacobi", "dtype": "float32", "points": 7, "nz": 512, "ny": 512, "nx": 512, "steps": 10},
        # a 27-offset stencil of shifted views, compiled once and applied
        {"name": "stencil_27", "kind": "stencil", "points": 27, "nz": 384, "ny": 512, "nx": 512},
        # weighted 2-D histogram of clustered points into the 1024 x 1024 configuration
        {"name": "hist_weighted", "kind": "hist", "points": 1 << 26, "nbx": 1024, "nby": 1024, "weighted": True},
        # uneven arrays, half float32 and half bfloat16: sum, mean, max, sum(x*x - x) of each in one call
        {"name": "batch_fixed", "kind": "batch", "arrays": 2000},
        # the same through the general form: any tapes and reductions per array
        {"name": "batch_general", "kind": "batch_expr", "arrays": 600, "outs": 4, "dtype": "mixed"},
        # pixel binning of an image on disjoint panels (the reference's benchmark, 2 x 2 x 2)
        {"name": "binning_panels", "kind": "binning", "form": "panels", "factor": 2, "n": 64, "h": 1024, "w": 1024},
        # a plain axis reduction
        {"name": "sum_axis0", "kind": "reduce", "op": "sum", "dtype": "float32", "n0": 4096, "n1": 1, "n2": 16384, "axis": 0},
        # dest[idx[i]] += src[i]
        {"name": "scatter_add", "kind": "scatter", "dtype": "float32", "n": 1 << 26, "entries": 1 << 20},
    ]


# ---- drawn cases -------------------------------------------------------------------------------------------------
def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["expr", "expr_reduce", "views", "frames", "jacobi", "stencil", "hist", "batch", "batch_expr", "binning",
                       "reduce", "scatter"])
    c = {"kind": kind}
    if kind == "expr":
        c.update(dtype=rng.choice(["float32", "float64", "bfloat16"]), h=_log(rng, 8, 4096), w=_log(rng, 16, 4096))
    elif kind == "expr_reduce":
        c.update(dtype=rng.choice(["float64", "float64", "float32"]), n0=_log(rng, 8, 256), n1=_log(rng, 16, 256),
                 n2=_log(rng, 16, 256))
    elif kind == "views":
        c.update(q=rng.choice([4, 5, 8, 16]), b=_log(rng, 16, 256), r=8 * _log(rng, 2, 32), p=rng.choice([32, 64, 77, 96, 128]))
    elif kind == "frames":
        n, h, w = _log(rng, 4, 128), _log(rng, 64, 1024), _log(rng, 64, 1100)
        y0, x0 = rng.randrange(0, h // 4), rng.randrange(0, w // 4)
        c.update(raw=rng.choice(["uint16", "float32", "int32"]), out=rng.choice(["float32", "float32", "bfloat16"]), n=n, h=h, w=w,
                 y0=y0, y1=rng.randrange(h // 2, h + 1), x0=x0, x1=rng.randrange(w // 2, w + 1))
    elif kind == "jacobi":
        f64 = rng.random() < 0.3   # float64 grids are smaller: the card's float64 rate is low
        c.update(dtype="float64" if f64 else "float32", points=rng.choice([7, 27]), nz=_log(rng, 24, 128 if f64 else 480),
                 ny=_log(rng, 32, 160 if f64 else 480), nx=rng.choice([1, 4, 4, 4]) * _log(rng, 16, 60 if f64 else 120),
                 steps=rng.randint(1, 4 if f64 else 10))
    elif kind == "stencil":
        c.update(points=rng.choice([7, 27]), nz=_log(rng, 24, 384), ny=_log(rng, 32, 480), nx=_log(rng, 32, 500))
    elif kind == "hist":
        c.update(points=_log(rng, 1 << 14, 1 << 26), nbx=_log(rng, 64, 1500), nby=_log(rng, 64, 1500), weighted=rng.random() < 0.5)
    elif kind == "batch":
        c.update(arrays=_log(rng, 20, 1800))
    elif kind == "batch_expr":
        c.update(arrays=_log(rng, 20, 600), outs=rng.randint(1, 4), dtype=rng.choice(["mixed", "float32", "float64", "int32"]))
    elif kind == "binning":
        c.update(form=rng.choice(["views", "panels", "reshape"]), factor=rng.choice([2, 2, 3, 4]), n=_log(rng, 8, 64),
                 h=_log(rng, 64, 1024), w=_log(rng, 64, 1024))
    elif kind == "reduce":
        c.update(op=rng.choice(["sum", "mean", "max", "argmax"]), dtype=rng.choice(["float32", "bfloat16", "float64", "int32"]),
                 n0=_log(rng, 4, 1024), n1=_log(rng, 4, 256), n2=_log(rng, 8, 512), axis=rng.choice([0, 1, 2, -1]))
    else:
        c.update(dtype=rng.choice(["float32", "float64", "int32"]), n=_log(rng, 1 << 14, 1 << 26), entries=_log(rng, 1 << 6, 1 << 22))
    return c


# ---- inputs ------------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 13)


def _dev(t, dtype):
    """A device array holding the torch tensor's values."""
    a = nca.NCDevArray(tuple(t.shape), nca.DType[dtype])
    _torch(a, dtype).copy_(t)
    return a


def _torch(a, dtype):
    """The torch view of a contiguous device array's memory."""
    n = a.size * _SIZE.get(dtype, 8)
    return a._buf[a._offset:a._offset + n].view(_T[dtype]).view(a.shape)


def _values(g, shape, dtype):
    if dtype in ("int32", "uint16"):
        return torch.randint(0 if dtype == "uint16" else -1000, 4000, shape, generator=g, device="cuda", dtype=torch.int32)
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.float64 if dtype == "float64" else torch.float32)


def _lengths(case, seed, most):
    rng = np.random.default_rng(int(seed) + 4)
    return np.round(np.exp(rng.uniform(np.log(64), np.log(most), case["arrays"]))).astype(np.int64)


def _uneven(case, seed, dtypes, most=1 << 22):
    """1-D arrays of log-uniform lengths, the i-th of type dtypes[i % len]: views into one buffer per type."""
    g, lens = _gen(seed), _lengths(case, seed, most)
    arrays, tensors = [None] * len(lens), [None] * len(lens)
    for k, dt in enumerate(dtypes):
        mine = range(k, len(lens), len(dtypes))
        total = int(sum(int(lens[i]) for i in mine))
        if dt == "int32":
            flat = torch.randint(-1000, 1000, (max(total, 1),), generator=g, device="cuda", dtype=torch.int32)
        else:
            flat = torch.exp(torch.randn(max(total, 1), generator=g, device="cuda") * 2.0)
            flat *= torch.where(torch.rand(flat.shape, generator=g, device="cuda") < 0.5, -1.0, 1.0)
            flat = flat.to(_T[dt])
        buf, at, size = flat.view(torch.uint8), 0, _SIZE[dt]
        for i in mine:
            n = int(lens[i])
            arrays[i] = nca.NCDevArray((n,), nca.DType[dt], _buf=buf, _offset=at * size)
            tensors[i] = flat[at:at + n]
            at += n
    return arrays, tensors


def _outs(case):
    """The outputs of a general batch: (function of the element, reduction)."""
    if case["dtype"] == "int32":   # batched outputs are floating
        half = lambda x: x * 0.5  # noqa: E731
        every = [(half, nca.RedOp.SUM), (half, nca.RedOp.MEAN), (half, nca.RedOp.MAX), (lambda x: x * 0.25, nca.RedOp.SUM)]
    else:
        every = [(None, nca.RedOp.SUM), (None, nca.RedOp.MEAN), (None, nca.RedOp.MAX), (lambda x: x * x - x, nca.RedOp.SUM)]
    return every[:case["outs"]]


def _stencil_weights(points):
    return laplacian7() if points == 7 else laplacian27()


def _used(points):
    w = _stencil_weights(points).reshape(27)
    return [(t, (t // 9, (t // 3) % 3, t % 3), float(w[t])) for t in range(27) if w[t] != 0.0]


_RED = {"sum": nca.RedOp.SUM, "mean": nca.RedOp.MEAN, "max": nca.RedOp.MAX, "argmax": nca.RedOp.ARGMAX}
_RED_OUT = {"sum": None, "mean": "float64", "max": None, "argmax": "int64"}


def _red_dtype(case):
    dt = _RED_OUT[case["op"]] or case["dtype"]
    return "float32" if dt == "bfloat16" else dt


def _points(case, g):
    """Points of a mixture of 8 Gaussians in the unit square, some outside it, and lognormal weights."""
    n = case["points"]
    centres = torch.rand((8, 2), generator=g, device="cuda")
    sigma = torch.rand(8, generator=g, device="cuda") * 0.09 + 0.01
    edges = torch.cumsum(torch.softmax(torch.randn(8, generator=g, device="cuda"), 0), 0)
    comp = torch.bucketize(torch.rand(n, generator=g, device="cuda"), edges).clamp_(max=7)
    s = sigma[comp]
    x = centres[:, 0][comp] + torch.randn(n, generator=g, device="cuda") * s
    y = centres[:, 1][comp] + torch.randn(n, generator=g, device="cuda") * s
    w = torch.exp(torch.randn(n, generator=g, device="cuda")) if case["weighted"] else None
    return x, y, w


def _inputs(case, seed):
    """The torch tensors of a case's inputs (what exact() computes from)."""
    g, k = _gen(seed), case["kind"]
    if k == "expr":
        return [_values(g, (case["h"], case["w"]), case["dtype"]).to(_T[case["dtype"]]) for _ in range(3)]
    if k == "expr_reduce":
        return [_values(g, (case["n0"], case["n1"], case["n2"]), case["dtype"]) for _ in range(3)]
    if k == "views":
        q, b, r, p = case["q"], case["b"], case["r"], case["p"]
        return [torch.randn((p, b, r, q), generator=g, device="cuda"), torch.randn((b,), generator=g, device="cuda"),
                torch.randint(-1000, 1001, (q, b, r, p), generator=g, device="cuda", dtype=torch.int32)]
    if k == "frames":
        n, h, w = case["n"], case["h"], case["w"]
        return [_values(g, (n, h, w), case["raw"]), 100 + torch.randn((h, w), generator=g, device="cuda"),
                1 + 0.1 * torch.randn((h, w), generator=g, device="cuda")]
    if k == "jacobi":
        return [_values(g, (case["nz"], case["ny"], case["nx"]), case["dtype"])]
    if k == "stencil":
        pad = torch.zeros((case["nz"] + 2, case["ny"] + 2, case["nx"] + 2), device="cuda")
        pad[1:-1, 1:-1, 1:-1] = torch.randn((case["nz"], case["ny"], case["nx"]), generator=g, device="cuda")
        return [pad]
    if k == "hist":
        return list(_points(case, g))
    if k == "binning":
        return [torch.rand((case["n"], case["h"], case["w"]), generator=g, device="cuda")]
    if k == "reduce":
        return [_values(g, (case["n0"], case["n1"], case["n2"]), case["dtype"]).to(_T[case["dtype"]])]
    if k == "scatter":
        src = _values(g, (case["n"],), case["dtype"])
        idx = torch.randint(0, case["entries"], (case["n"],), generator=g, device="cuda", dtype=torch.int32)
        return [idx, src]
    raise ValueError(k)


def prepare(case, seed):
    k = case["kind"]
    st = {"case": case, "kind": k}
    if k == "batch":
        arrays, _ = _uneven(case, seed, ["float32", "bfloat16"])
        st["batch"] = Batch(arrays)
        st["res"] = _torch(st["batch"].results, "float64")
        return st
    if k == "batch_expr":
        dts = ["float32", "bfloat16"] if case["dtype"] == "mixed" else [case["dtype"]]
        arrays, _ = _uneven(case, seed, dts)
        outs = _outs(case)
        st["batch"] = BatchExpr([(a, outs) for a in arrays])
        st["res"] = st["batch"].results._buf.view(torch.float64).view(-1, 4, 2)[:case["arrays"]]
        return st
    t = _inputs(case, seed)
    if k == "expr":
        st["a"], st["b"], st["c"] = (_dev(x, case["dtype"]) for x in t)
        st["dtype"] = "float32" if case["dtype"] == "bfloat16" else case["dtype"]
    elif k == "expr_reduce":
        a, b, c = (_dev(x, case["dtype"]) for x in t)
        with nca.lazy_mode():
            st["e"] = a * b + nca.sqrt(abs(c)) - 0.5 * a
        st["out"] = nca.NCDevArray(st["e"].shape, st["e"].dtype)
        plane = (case["n1"], case["n2"])
        st["s"], st["m"] = nca.NCDevArray(plane, st["e"].dtype), nca.NCDevArray(plane, st["e"].dtype)
        st["ts"], st["tm"] = nca.NCDevArray((), st["e"].dtype), nca.NCDevArray((), st["e"].dtype)
        st["es"], st["em"] = nca.DevExpr.leaf(st["s"]), nca.DevExpr.leaf(st["m"])
        st["res"] = [_torch(st[n], case["dtype"]) for n in ("out", "s", "m", "ts", "tm")]
    elif k == "views":
        x, v, kk = _dev(t[0], "float32"), _dev(t[1], "float32"), _dev(t[2], "int32")
        with nca.lazy_mode():
            st["y"] = x.permute(3, 1, 2, 0) * v.reshape(1, case["b"], 1, 1) + kk
            st["z"] = (kk * 3 + 7) % 11
        st["yo"], st["zo"] = nca.NCDevArray(st["y"].shape, st["y"].dtype), nca.NCDevArray(st["z"].shape, st["z"].dtype)
        kept = (case["q"], case["b"], case["p"])
        st["mx"], st["am"] = nca.NCDevArray(kept, nca.DType.float32), nca.NCDevArray(kept, nca.DType.int64)
        st["res"] = [_torch(st["yo"], "float32"), _torch(st["zo"], "int32"), _torch(st["mx"], "float32"), _torch(st["am"], "int64")]
    elif k == "frames":
        y, x = slice(case["y0"], case["y1"]), slice(case["x0"], case["x1"])
        raw = _dev(t[0].to(_T[case["raw"]]), case["raw"])[:, y, x]
        dark, gain = _dev(t[1], "float32")[y, x], _dev(t[2], "float32")[y, x]
        with nca.lazy_mode():
            st["e"] = (raw - dark) * gain
        st["out"] = nca.NCDevArray(st["e"].shape, nca.DType[case["out"]])
        st["res"] = _torch(st["out"], case["out"])
    elif k == "jacobi":
        st["st"] = Stencil3D(_stencil_weights(case["points"]), 0.1)
        st["a"] = _dev(t[0], case["dtype"])
        st["b"] = nca.NCDevArray(st["a"].shape, st["a"].dtype)
        st["res"] = _torch(st["a"] if case["steps"] % 2 == 0 else st["b"], case["dtype"])
    elif k == "stencil":
        used = _used(case["points"])
        centre = [i for i, u in enumerate(used) if u[0] == 13][0]

        def lap(views):
            acc = None
            for v, (_, _, w) in zip(views, used):
                term = nca.DevExpr.leaf(v) * np.float32(w)
                acc = term if acc is None else acc + term
            return nca.DevExpr.leaf(views[centre]) + acc * np.float32(0.1)

        st["st"] = Stencil.create([u[1] for u in used], lap, nca.DType.float32)
        st["src"] = _dev(t[0], "float32")
        st["dst"] = nca.NCDevArray((case["nz"], case["ny"], case["nx"]), nca.DType.float32)
        st["res"] = _torch(st["dst"], "float32")
    elif k == "hist":
        st["x"], st["y"] = _dev(t[0], "float32"), _dev(t[1], "float32")
        st["w"] = _dev(t[2], "float32") if case["weighted"] else None
    elif k == "binning":
        f = case["factor"]
        n, h, w = (e // f for e in (case["n"], case["h"], case["w"]))
        data = _dev(t[0], "float32")
        st["out"] = nca.NCDevArray((n, h, w), nca.DType.float32)
        st["res"] = _torch(st["out"], "float32")
        if case["form"] == "reshape":
            crop = data[:n * f, :h * f, :w * f]
            st["e"] = nca.DevExpr.leaf(crop.reshape(n, f, h, f, w, f))
        else:
            if case["form"] == "panels":
                data = nca.NCDevArray.from_panels([data[i].copy() for i in range(case["n"])])
            e = None
            with nca.lazy_mode():
                for a in range(f):
                    for b in range(f):
                        for c in range(f):
                            v = data[a:a + (n - 1) * f + 1:f, b:b + (h - 1) * f + 1:f, c:c + (w - 1) * f + 1:f]
                            e = v if e is None else e + v
                st["e"] = e * (1.0 / f ** 3)
    elif k == "reduce":
        x = _dev(t[0], case["dtype"])
        if case["n1"] == 1:
            x = x.reshape(case["n0"], case["n2"])
        st["e"] = nca.DevExpr.leaf(x)
        st["red"] = [(_RED[case["op"]], None if case["axis"] < 0 else case["axis"])]
        st["dtype"] = _red_dtype(case)
    elif k == "scatter":
        st["idx"], st["src"] = _dev(t[0], "int32"), _dev(t[1], case["dtype"])
        st["dest"] = nca.NCDevArray((case["entries"],), nca.DType[case["dtype"]])
        st["res"] = _torch(st["dest"], case["dtype"])
    return st


# ---- one pass ----------------------------------------------------------------------------------------------------
def run(st):
    k = st["kind"]
    if k == "expr":
        a = st["a"]
        with nca.lazy_mode():
            e = a * st["b"] + nca.sqrt(abs(st["c"])) - 0.5 * a
        return _torch(e.materialize(), st["dtype"])
    if k == "expr_reduce":
        st["e"].evaluate(out=st["out"], reductions=[(nca.RedOp.SUM, 0), (nca.RedOp.MAX, 0)], red_out=[st["s"], st["m"]])
        st["es"].evaluate(reductions=[(nca.RedOp.SUM, None)], red_out=[st["ts"]])
        st["em"].evaluate(reductions=[(nca.RedOp.MAX, None)], red_out=[st["tm"]])
        return st["res"]
    if k == "views":
        nca.evaluate_many([(st["y"], st["yo"]), (st["z"], st["zo"])], reductions=[(nca.RedOp.MAX, 2), (nca.RedOp.ARGMAX, 2)],
                          red_out=[st["mx"], st["am"]])
        return st["res"]
    if k == "frames":
        st["e"].evaluate(out=st["out"])
        return st["res"]
    if k == "jacobi":
        st["st"].iterate(st["a"], st["b"], st["case"]["steps"])
        return st["res"]
    if k == "stencil":
        st["st"].apply(st["src"], st["dst"])
        return st["res"]
    if k == "hist":
        c = st["case"]
        counts, wsum = hist2d(st["x"], st["y"], c["nbx"], c["nby"], w=st["w"])
        return [_torch(counts, "int64"), _torch(wsum, "float32") if wsum is not None else None]
    if k == "batch":
        st["batch"].run(graph=True)
        return [st["res"][:, i] for i in range(4)]
    if k == "batch_expr":
        st["batch"].launch(graph=True)
        return [st["res"][:, i, 0] for i in range(st["case"]["outs"])]
    if k == "binning":
        if st["case"]["form"] == "reshape":
            st["e"].evaluate(reductions=[(nca.RedOp.SUM, (1, 3, 5))], red_out=[st["out"]])
        else:
            st["e"].evaluate(out=st["out"])
        return st["res"]
    if k == "reduce":
        (r,) = st["e"].evaluate(reductions=st["red"])
        return _torch(r, st["dtype"])
    st["dest"].fill(0)
    st["dest"].scatter_add(st["idx"], st["src"])
    return st["res"]


# ---- what a pass cannot do without -------------------------------------------------------------------------------
def work(case):
    k = case["kind"]
    if k == "expr":
        n, s = case["h"] * case["w"], _SIZE[case["dtype"]]
        return {"bytes": n * (3 * s + max(s, 4)), "flops": 6 * n}
    if k == "expr_reduce":
        s, n, plane = _SIZE[case["dtype"]], case["n0"] * case["n1"] * case["n2"], case["n1"] * case["n2"]
        return {"bytes": s * (4 * n + 2 * plane + 2), "flops": 8 * n}
    if k == "views":
        n, kept = case["q"] * case["b"] * case["r"] * case["p"], case["q"] * case["b"] * case["p"]
        return {"bytes": 16 * n + 12 * kept + 4 * case["b"], "flops": 6 * n}
    if k == "frames":
        plane = (case["y1"] - case["y0"]) * (case["x1"] - case["x0"])
        return {"bytes": plane * (case["n"] * (_SIZE[case["raw"]] + _SIZE[case["out"]]) + 8), "flops": 2 * plane * case["n"]}
    if k == "jacobi":
        n = case["nz"] * case["ny"] * case["nx"]
        return {"bytes": 2 * n * _SIZE[case["dtype"]], "flops": 2 * n * (case["points"] + 1) * case["steps"]}
    if k == "stencil":
        n = case["nz"] * case["ny"] * case["nx"]
        return {"bytes": 4 * n + 4 * (case["nz"] + 2) * (case["ny"] + 2) * (case["nx"] + 2), "flops": 2 * n * (case["points"] + 1)}
    if k == "hist":
        bins = case["nbx"] * case["nby"]
        return {"bytes": (12 if case["weighted"] else 8) * (case["points"] + bins), "flops": 4 * case["points"]}
    if k in ("batch", "batch_expr"):
        # lengths are log-uniform: their mean over the distribution
        mean = ((1 << 22) - 64) / math.log((1 << 22) / 64)
        size = {"float32": 4, "float64": 8, "int32": 4}.get(case.get("dtype"), 3)
        return {"bytes": case["arrays"] * (mean * size + 32), "flops": 4 * case["arrays"] * mean}
    if k == "binning":
        n = math.prod(case[e] // case["factor"] for e in ("n", "h", "w"))
        return {"bytes": 4 * n * (case["factor"] ** 3 + 1), "flops": n * case["factor"] ** 3}
    if k == "reduce":
        n = case["n0"] * case["n1"] * case["n2"]
        kept = 1 if case["axis"] < 0 else n // (case["n2"] if case["n1"] == 1 and case["axis"] == 1 else case["n%d" % case["axis"]])
        return {"bytes": n * _SIZE[case["dtype"]] + kept * _SIZE[_red_dtype(case)], "flops": n}
    return {"bytes": case["n"] * (4 + _SIZE[case["dtype"]]) + case["entries"] * _SIZE[case["dtype"]], "flops": case["n"]}


# ---- the outputs in 64 bits --------------------------------------------------------------------------------------
def _laplace(u, points, shape):
    """sum_o w_o u[c + o] of a padded grid, 64 bits."""
    acc = torch.zeros(shape, device="cuda", dtype=torch.float64)
    for _, (z, y, x), w in _used(points):
        acc.add_(u[z:z + shape[0], y:y + shape[1], x:x + shape[2]], alpha=w)
    return acc


def exact(case, seed):
    k = case["kind"]
    if k == "batch":
        _, tensors = _uneven(case, seed, ["float32", "bfloat16"])
        rows = []
        for t in tensors:
            d = t.double()
            s = d.sum()
            rows.append(torch.stack([s, s / d.numel(), d.max(), (d * d - d).sum()]))
        m = torch.stack(rows)
        return [m[:, i] for i in range(4)]
    if k == "batch_expr":
        dts = ["float32", "bfloat16"] if case["dtype"] == "mixed" else [case["dtype"]]
        _, tensors = _uneven(case, seed, dts)
        rows = []
        for t in tensors:
            d = t.double()
            if case["dtype"] == "int32":
                s = d.sum() * 0.5
                rows.append(torch.stack([s, s / d.numel(), d.max() * 0.5, d.sum() * 0.25]))
            else:
                s = d.sum()
                rows.append(torch.stack([s, s / d.numel(), d.max(), (d * d - d).sum()]))
        m = torch.stack(rows)
        return [m[:, i] for i in range(case["outs"])]
    t = _inputs(case, seed)
    if k == "expr":
        a, b, c = (x.double() for x in t)
        return a * b + c.abs().sqrt() - 0.5 * a
    if k == "expr_reduce":
        a, b, c = (x.double() for x in t)
        y = a * b + c.abs().sqrt() - 0.5 * a
        s, m = y.sum(0), y.amax(0)
        return [y, s, m, s.sum(), m.max()]
    if k == "views":
        y = t[0].double().permute(3, 1, 2, 0) * t[1].double().view(1, -1, 1, 1) + t[2].double()
        return [y.contiguous(), None, y.amax(2), None]
    if k == "frames":
        y, x = slice(case["y0"], case["y1"]), slice(case["x0"], case["x1"])
        return (t[0][:, y, x].double() - t[1][y, x].double()) * t[2][y, x].double()
    if k == "jacobi":
        shape = tuple(t[0].shape)
        u = torch.zeros([e + 2 for e in shape], device="cuda", dtype=torch.float64)
        core = u[1:-1, 1:-1, 1:-1]
        core.copy_(t[0])
        for _ in range(case["steps"]):
            core.add_(_laplace(u, case["points"], shape), alpha=0.1)
        return core.contiguous()
    if k == "stencil":
        u = t[0].double()
        return u[1:-1, 1:-1, 1:-1] + 0.1 * _laplace(u, case["points"], (case["nz"], case["ny"], case["nx"]))
    if k == "hist":
        if not case["weighted"]:
            return None
        x, y, w = t
        ix, iy = torch.floor(x * float(case["nbx"])), torch.floor(y * float(case["nby"]))   # the bins are defined in float32
        ok = (ix >= 0) & (ix < case["nbx"]) & (iy >= 0) & (iy < case["nby"])
        cell = (iy[ok].long() * case["nbx"] + ix[ok].long())
        return [None, torch.zeros(case["nbx"] * case["nby"], device="cuda", dtype=torch.float64)
                .index_add_(0, cell, w[ok].double()).view(case["nby"], case["nbx"])]
    if k == "binning":
        f = case["factor"]
        n, h, w = (e // f for e in (case["n"], case["h"], case["w"]))
        s = t[0][:n * f, :h * f, :w * f].double().reshape(n, f, h, f, w, f).sum((1, 3, 5))
        return s if case["form"] == "reshape" else s / f ** 3
    if k == "reduce":
        if case["op"] == "argmax" or (case["dtype"] == "int32" and case["op"] != "mean"):
            return None
        x = t[0].double()
        if case["n1"] == 1:
            x = x.reshape(case["n0"], case["n2"])
        axis = tuple(range(x.ndim)) if case["axis"] < 0 else case["axis"]
        return {"sum": torch.sum, "mean": torch.mean, "max": torch.amax}[case["op"]](x, axis)
    if case["dtype"] == "int32":
        return None
    return torch.zeros(case["entries"], device="cuda", dtype=torch.float64).index_add_(0, t[0].long(), t[1].double())
