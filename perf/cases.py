"""What a user of this framework has it do, as cases that can be timed.

A case is a dict of plain values.  `prepare` makes a case's arrays on the GPU
and lowers its expressions (what a caller of the C ABI does once), `run` makes
the calls, `exact` gives the same results in 64 bits from plain torch, and
`work` counts the bytes and operations that the results need.

Arrays live in torch tensors, and every call goes through the C ABI on torch's
default stream with expressions lowered beforehand, as a C++ caller's
expressions are lowered when its call site is compiled.
"""
import ctypes as C
import math
import random

import numpy as np
import torch

import xtensor_gb300 as xg
from xtensor_gb300 import ops
from xtensor_gb300._ffi import check
from xtensor_gb300.batch import Batch
from xtensor_gb300.chunked import ChunkedArray, _sigs
from xtensor_gb300.device import DeviceArray
from xtensor_gb300.expr import lower

TORCH = {"float32": torch.float32, "float64": torch.float64, "bfloat16": torch.bfloat16, "int32": torch.int32,
         "int64": torch.int64, "bool": torch.bool}
SIZE = {"float32": 4, "float64": 8, "bfloat16": 2, "int32": 4, "int64": 8, "bool": 1}
EPS = 1e-5


def listed():
    """One case of each kind of work; `draw` spreads every kind over its range.

    The sizes come from the benchmark's workloads (2048 x 2048; 256 x 512 x
    1024; 2^28 elements; instances of 1..4096 rows of 16..2048 columns;
    requests from 1e3 elements up), and half of them are the same work at
    sizes that no vector width divides."""
    return [
        # the smallest calls: a stream of small requests of every expression
        # kind, each one or two launches: latency and launches count
        {"name": "requests_small", "kind": "requests", "mix": 11, "n": 16, "lo": 1000, "hi": 100000},
        # E = A*b + exp(-A*A) kept, and its row sums, in one call
        {"name": "fused_2048_f32", "kind": "fused", "rows": 2048, "cols": 2048, "dtype": "float32"},
        # many uneven instances of sum(A*v + C, {1}) in one batched launch
        {"name": "batch_rowsum_f32", "kind": "batch", "n": 256, "mix": 3, "max_rows": 4096, "max_cols": 2048},
        # a permuted copy of a large array
        {"name": "transpose_f32", "kind": "transpose", "d0": 256, "d1": 512, "d2": 1024, "perm": "201",
         "dtype": "float32"},
        # row normalisation (x - mean) / sqrt(var + eps), large and in double
        {"name": "normalize_f64", "kind": "normalize", "rows": 131072, "cols": 1024, "dtype": "float64"},
        # the same with rows that start at any element
        {"name": "normalize_odd_f32", "kind": "normalize", "rows": 60001, "cols": 777, "dtype": "float32"},
        # a reduction over the first and last axis
        {"name": "amax_02_f64", "kind": "reduce", "op": "amax", "axes": "02", "d0": 256, "d1": 512, "d2": 1024,
         "dtype": "float64"},
        # positions of the largest values along the middle axis, odd extents
        {"name": "argmax_odd_f32", "kind": "argmax", "axis": 1, "d0": 201, "d1": 399, "d2": 1001, "dtype": "float32"},
        # sum, mean, variance and norm of a whole array from one read
        {"name": "moments_bf16", "kind": "moments", "n": 1 << 28, "dtype": "bfloat16"},
        # a running sum over a whole array
        {"name": "cumsum_flat_f32", "kind": "cumsum", "axis": -1, "d0": 128, "d1": 512, "d2": 1024,
         "dtype": "float32"},
        # the elements above a threshold, compacted in order (the count comes
        # first: the caller sizes the result by it)
        {"name": "filter_f32", "kind": "views", "op": "filter", "n": 1 << 26, "dtype": "float32"},
        # a chunked array with edge chunks on every axis: assignment into the
        # chunks, then sums over the last axis
        {"name": "chunked_edges_f32", "kind": "chunked", "d0": 256, "d1": 512, "d2": 1024, "c0": 100, "c1": 200,
         "c2": 1000, "dtype": "float32"},
    ]


# ---- drawn cases ----------------------------------------------------------------------


def _log(rng, lo, hi):
    """An integer, log-uniform in [lo, hi]."""
    return int(min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _dims(rng, lo, hi):
    """Three extents of lo..hi elements altogether; one time in two the last
    is a multiple of 16, else any."""
    n = _log(rng, lo, hi)
    d2 = _log(rng, 16, min(2048, max(17, n // 4)))
    if rng.random() < 0.5:
        d2 = max(16, d2 // 16 * 16)
    d1 = _log(rng, 2, max(3, min(1024, n // d2)))
    return {"d0": max(1, n // (d1 * d2)), "d1": d1, "d2": d2}


def draw(rng):
    big = 1 << 27
    kind = rng.choice(["requests", "fused", "batch", "transpose", "normalize", "normalize", "reduce", "argmax",
                       "moments", "cumsum", "views", "chunked"])
    flt = rng.choice(["float32", "float32", "float64"])
    any_dt = rng.choice(["float32", "float32", "float64", "int32"])
    if kind == "requests":
        lo = _log(rng, 1000, 10000)
        return {"kind": kind, "mix": rng.randrange(1 << 20), "n": rng.randint(4, 24), "lo": lo,
                "hi": _log(rng, 2 * lo, 200 * lo)}
    if kind == "fused":
        cols = _log(rng, 16, 4096)
        return {"kind": kind, "rows": max(1, _log(rng, 10000, 1 << 25) // cols), "cols": cols, "dtype": flt}
    if kind == "batch":
        return {"kind": kind, "n": _log(rng, 16, 256), "mix": rng.randrange(1 << 20), "max_rows": _log(rng, 64, 4096),
                "max_cols": _log(rng, 64, 2048)}
    if kind == "transpose":
        return {"kind": kind, **_dims(rng, 100000, big if any_dt != "float64" else big // 2),
                "perm": rng.choice(["201", "210", "102", "021", "120"]), "dtype": any_dt}
    if kind == "normalize":
        cols = _log(rng, 16, 2048)
        if rng.random() < 0.4:
            cols = max(16, cols // 16 * 16)
        return {"kind": kind, "rows": max(1, _log(rng, 100000, big) // cols), "cols": cols, "dtype": flt}
    if kind == "reduce":
        op = rng.choice(["sum", "mean", "variance", "amax", "norm_l2"])
        return {"kind": kind, "op": op, "axes": rng.choice(["02", "0", "1", "2", "12", "01"]),
                **_dims(rng, 100000, big), "dtype": any_dt if op in ("sum", "amax") else flt}
    if kind == "argmax":
        return {"kind": kind, "axis": rng.choice([0, 1, 1, 2]), **_dims(rng, 100000, big), "dtype": any_dt}
    if kind == "moments":
        return {"kind": kind, "n": _log(rng, 100000, 1 << 28), "dtype": rng.choice(["float32", "bfloat16"])}
    if kind == "cumsum":
        return {"kind": kind, "axis": rng.choice([-1, -1, 0, 1, 2]), **_dims(rng, 100000, 1 << 26), "dtype": any_dt}
    if kind == "views":
        return {"kind": kind, "op": rng.choice(["filter", "filter", "filtration", "masked", "gather"]),
                "n": _log(rng, 100000, 1 << 26), "dtype": any_dt}
    d = _dims(rng, 1 << 20, big)
    cut = {"c%d" % i: max(8, -(-d["d%d" % i] // rng.randint(1, 4)) + rng.choice([0, 0, 1, 5])) for i in range(3)}
    return {"kind": "chunked", **d, **{k: min(v, d["d" + k[1]]) for k, v in cut.items()}, "dtype": flt}


# ---- arrays ---------------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _values(g, shape, dtype, scale=1.0):
    """Data as the workloads have it: N(0, 1) floats, integers of +-1000."""
    if dtype == "int32":
        return torch.randint(-1000, 1001, shape, generator=g, device="cuda", dtype=torch.int32)
    x = torch.randn(shape, generator=g, device="cuda", dtype=torch.float64 if dtype == "float64" else torch.float32)
    return (x * scale if scale != 1.0 else x).to(TORCH[dtype])


def _lognormal(g, n, dtype):
    """Sign-random lognormal(0, 2) magnitudes: 1e-6 .. 1e6."""
    x = torch.randn((n,), generator=g, device="cuda").mul_(2.0).exp_()
    x *= torch.randint(0, 2, (n,), generator=g, device="cuda", dtype=torch.int8).mul_(2).sub_(1)
    return x.to(TORCH[dtype])


def _empty(shape, dtype):
    return torch.zeros(shape, dtype=TORCH[dtype], device="cuda")


def _name(t):
    return {v: k for k, v in TORCH.items()}[t.dtype]


def _arr(t):
    """The framework's array over a torch tensor's memory."""
    return DeviceArray(tuple(t.shape), _name(t), t.data_ptr(), t.stride(), base=t)


class Call:
    """A call of the C ABI with its expression lowered: what a call site is."""

    def __init__(self, fn, exprs, *args):
        self.fn, self.keep, self.args = fn, [exprs], []
        for e in exprs:
            ex, leaves = lower(e)
            self.keep += [ex, leaves]
            self.args.append(C.byref(ex))
        for a in args:
            if isinstance(a, torch.Tensor):
                a = _arr(a)
            if isinstance(a, DeviceArray):
                self.keep.append(a)
                a = a.xtg_array()
            if isinstance(a, C.Structure):
                self.keep.append(a)
                a = C.byref(a)
            self.args.append(a)
        self.args.append(None)  # the default stream

    def __call__(self):
        check(self.fn(*self.args))


def _assign(out, e):
    return Call(xg.lib().xtg_assign, [e], out)


def _reduce(op, e, axes, out, **kw):
    return Call(xg.lib().xtg_reduce, [e], ops.make_desc(op, axes=axes, **kw), out)


def _argmax(e, axis, out):
    return Call(xg.lib().xtg_argreduce, [e], 0, 1, axis, out)


def _result(op, dtype):
    return "float64" if op in ("mean", "variance", "norm_l2") else dtype


def _c0(A, b):
    return A * b + xg.exp(-A * A)


def _normalized(x):
    return (x - xg.rmean(x)) / xg.sqrt(xg.rvar(x) + EPS)


# ---- the request mix ------------------------------------------------------------------


def _requests(case):
    """What each request of the mix is: (what, dtype, shape), the serving
    workload's kinds with float32 / float64 / int32 at 50 / 25 / 25 %."""
    r = random.Random("%d requests" % case["mix"])
    got = []
    for _ in range(case["n"]):
        n = int(round(math.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"])))))
        dt = r.choice(["float32", "float32", "float64", "int32"])
        what = r.choice(["c0", "c0sum", "affine", "full", "transpose", "normalize", "amax", "argmax"])
        if dt == "int32" and what in ("c0", "c0sum", "normalize"):
            what = r.choice(["affine", "full", "transpose"])
        cols = int(min(4096, max(16, 2 ** round(math.log2(n ** 0.5)))))
        if what == "full":
            shape = (n,)
        elif what in ("c0", "c0sum", "affine"):
            shape = (max(1, n // cols), cols)
        else:
            d1 = max(1, min(512, n // cols // 4))
            shape = (max(1, n // (d1 * cols)), d1, cols)
        got.append((what, dt, shape))
    return got


def _request(what, dt, shape, g):
    """(inputs, calls, outputs) of one request."""
    x = _values(g, shape, dt)
    a = _arr(x)
    if what in ("c0", "c0sum"):
        b = _values(g, shape[-1:], dt)
        e = _c0(a, _arr(b))
        out = _empty(shape if what == "c0" else shape[:1], dt)
        return [x, b], [_assign(out, e) if what == "c0" else _reduce("sum", e, [1], out)], out
    if what == "affine":
        v, c = _values(g, shape[-1:], dt), _values(g, shape, dt)
        out = _empty(shape[:1], dt)
        return [x, v, c], [_reduce("sum", a * _arr(v) + _arr(c), [1], out)], out
    if what == "full":
        op = "sum" if dt == "int32" else "variance"
        out = _empty((), _result(op, dt))
        return [x], [_reduce(op, a, None, out)], out
    if what == "transpose":
        out = _empty((shape[2], shape[0], shape[1]), dt)
        return [x], [_assign(out, a.transpose((2, 0, 1)))], out
    if what == "normalize":
        out = _empty(shape, dt)
        return [x], [_assign(out, _normalized(a))], out
    if what == "amax":
        out = _empty((shape[1],), dt)
        return [x], [_reduce("amax", a, [0, 2], out)], out
    out = _empty((shape[0], shape[2]), "int32")
    return [x], [_argmax(a, 1, out)], out


def _request_exact(what, dt, ins):
    d = [t.double() for t in ins]
    x = d[0]
    if what in ("c0", "c0sum"):
        e = x * d[1] + torch.exp(-x * x)
        return e if what == "c0" else e.sum(1)
    if what == "affine":
        return (x * d[1] + d[2]).sum(1)
    if what == "full":
        return x.sum() if dt == "int32" else x.var(correction=0)
    if what == "transpose":
        return x.permute(2, 0, 1).contiguous()
    if what == "normalize":
        return (x - x.mean(2, keepdim=True)) / torch.sqrt(x.var(2, correction=0, keepdim=True) + EPS)
    return x.amax((0, 2)) if what == "amax" else None


def _request_bytes(what, dt, shape):
    s, n = SIZE[dt], math.prod(shape)
    return {"c0": 2 * n * s + shape[-1] * s, "c0sum": n * s + (shape[-1] + shape[0]) * s,
            "affine": 2 * n * s + (shape[-1] + shape[0]) * s, "full": n * s + 8, "transpose": 2 * n * s,
            "normalize": 2 * n * s, "amax": n * s + shape[1 % len(shape)] * s,
            "argmax": n * s + shape[0] * shape[-1] * 4}[what]


# ---- batched instances ----------------------------------------------------------------


def _instances(case):
    """(rows, cols) of each instance: both uniform, as in the batching workload."""
    r = np.random.default_rng(case["mix"])
    rows = r.integers(1, case["max_rows"] + 1, case["n"])
    cols = r.integers(16, case["max_cols"] + 1, case["n"])
    return [(int(a), int(b)) for a, b in zip(rows, cols)]


def _carve(slab, at, shape):
    """A tensor of `shape` in the slab from element `at` on, and the next
    256-byte aligned place after it."""
    n = math.prod(shape)
    return slab[at:at + n].view(shape), at + -(-n // 64) * 64


def _batch_arrays(case, seed):
    """One slab holds every instance's A and C, one every v, one every result."""
    g = _gen(seed)
    sizes = _instances(case)
    up = lambda n: -(-n // 64) * 64  # noqa: E731
    big = torch.rand((sum(2 * up(r * c) for r, c in sizes),), generator=g, device="cuda").mul_(2.0).sub_(1.0)
    vec = torch.randn((sum(up(c) for _, c in sizes),), generator=g, device="cuda")
    res = _empty((sum(up(r) for r, _ in sizes),), "float32")
    a = v = o = 0
    inst = []
    for r, c in sizes:
        A, a = _carve(big, a, (r, c))
        Cm, a = _carve(big, a, (r, c))
        b, v = _carve(vec, v, (c,))
        out, o = _carve(res, o, (r,))
        inst.append((A, b, Cm, out))
    return inst, res


# ---- chunked arrays -------------------------------------------------------------------


def _chunk_grid(case):
    """(shape, chunk shape, bytes between chunks, [(slices, extents) by chunk])."""
    shape = tuple(case["d%d" % i] for i in range(3))
    cs = tuple(case["c%d" % i] for i in range(3))
    per = -(-math.prod(cs) * SIZE[case["dtype"]] // 256) * 256 // SIZE[case["dtype"]]
    grid = [-(-s // c) for s, c in zip(shape, cs)]
    cells = []
    for i in range(grid[0]):
        for j in range(grid[1]):
            for k in range(grid[2]):
                at = [(q * c, min((q + 1) * c, s)) for q, c, s in zip((i, j, k), cs, shape)]
                cells.append((tuple(slice(*t) for t in at), tuple(t[1] - t[0] for t in at)))
    return shape, cs, per, cells


# ---- prepare / run --------------------------------------------------------------------


def _shape(case):
    return (case["d0"], case["d1"], case["d2"])


def _axes(case):
    return [int(a) for a in case["axes"]]


def prepare(case, seed):
    xg.init(0)
    L = xg.lib()
    kind, g = case["kind"], _gen(seed)
    dt = case.get("dtype", "float32")
    if kind == "requests":
        parts = [_request(*r, g) for r in _requests(case)]
        return {"calls": [c for _, cs, _ in parts for c in cs], "out": [o for _, _, o in parts],
                "in": [i for i, _, _ in parts]}
    if kind == "fused":
        A = torch.rand((case["rows"], case["cols"]), generator=g, device="cuda", dtype=TORCH[dt]).mul_(2).sub_(1)
        b = _values(g, (case["cols"],), dt)
        E, r = _empty(A.shape, dt), _empty((case["rows"],), dt)
        call = Call(L.xtg_assign_reduce, [_c0(_arr(A), _arr(b))], E, ops.make_desc("sum", axes=[1]), r)
        return {"in": [A, b], "calls": [call], "out": [E, r]}
    if kind == "batch":
        inst, res = _batch_arrays(case, seed)
        tree = [(_arr(A) * _arr(v) + _arr(Cm), _arr(o)) for A, v, Cm, o in inst]
        b = Batch(tree[0][0], reduce="sum")
        for e, o in tree:
            b.add(e, o)
        b.build(autotune=True)
        return {"in": inst, "calls": [b.run], "out": [res]}
    if kind == "transpose":
        x = _values(g, _shape(case), dt)
        perm = tuple(int(c) for c in case["perm"])
        out = _empty([x.shape[p] for p in perm], dt)
        return {"in": [x], "calls": [_assign(out, _arr(x).transpose(perm))], "out": [out]}
    if kind == "normalize":
        x = _values(g, (case["rows"], case["cols"]), dt)
        out = _empty(x.shape, dt)
        return {"in": [x], "calls": [_assign(out, _normalized(_arr(x)))], "out": [out]}
    if kind == "reduce":
        x, axes = _values(g, _shape(case), dt), _axes(case)
        out = _empty([n for i, n in enumerate(x.shape) if i not in axes], _result(case["op"], dt))
        return {"in": [x], "calls": [_reduce(case["op"], _arr(x), axes, out)], "out": [out]}
    if kind == "argmax":
        x = _values(g, _shape(case), dt)
        out = _empty([n for i, n in enumerate(x.shape) if i != case["axis"]], "int32")
        return {"in": [x], "calls": [_argmax(_arr(x), case["axis"], out)], "out": [out]}
    if kind == "moments":
        x = _lognormal(g, case["n"], dt)
        outs = [_empty((), "float32")] + [_empty((), "float64") for _ in range(3)]
        call = Call(L.xtg_reduce_moments, [_arr(x)], ops.make_desc("variance"), *outs)
        return {"in": [x], "calls": [call], "out": outs}
    if kind == "cumsum":
        x = _values(g, _shape(case), dt)
        ax = case["axis"]
        out = _empty(x.shape if ax >= 0 else (x.numel(),), dt)
        return {"in": [x], "calls": [Call(L.xtg_accumulate, [_arr(x)], 0, int(ax >= 0), max(ax, 0), -1, out)],
                "out": [out]}
    if kind == "views":
        return _prepare_views(case, g, L)
    # chunked: the expression into every chunk, then sums over the last axis
    shape, cs, per, cells = _chunk_grid(case)
    x = _values(g, shape, dt)
    slab = _empty((per * len(cells),), dt)
    whole = DeviceArray((slab.numel(),), dt, slab.data_ptr(), base=slab)
    chunks = [DeviceArray(cs, dt, slab.data_ptr() + i * per * SIZE[dt], base=whole) for i in range(len(cells))]
    ch = ChunkedArray(shape, cs, dt, chunks=chunks)
    rows = _empty(shape[:2], dt)
    cl = (C.c_void_p * 1)()  # no operand of the assignment is chunked itself
    to, rd, ro = ch.xtg_chunked(), ops.make_desc("sum", axes=[2]), _arr(rows).xtg_array()
    ex, leaves = lower(_arr(x) * 2.0 + 1.0)
    f = _sigs()

    def assign():
        check(f.xtg_chunked_assign(C.addressof(ex), C.addressof(cl), C.byref(to), None))

    def sums():
        check(f.xtg_chunked_reduce(C.byref(to), C.byref(rd), C.byref(ro), None))

    return {"in": [x, ch, leaves], "calls": [assign, sums], "out": [slab, rows]}


def _prepare_views(case, g, L):
    n, dt, op = case["n"], case["dtype"], case["op"]
    x = _values(g, (n,), dt)
    one = 1000 * 0.5 if dt == "int32" else 1.0
    cond = _arr(x) > (int(one) if dt == "int32" else one)
    if op == "filter":
        out, count = _empty((n,), dt), C.c_int64()
        ask = Call(L.xtg_filter_count, [cond], C.byref(count))
        (vx, vk), (cx, ck) = lower(xg.leaf(_arr(x))), lower(cond)

        def read():
            ask()
            o = _arr(out[:count.value]).xtg_array()
            check(L.xtg_filter(C.byref(vx), C.byref(cx), C.byref(o), None))
            return [out, count.value]

        return {"in": [x, vk, ck], "read": read}
    z = _values(g, (n,), dt)
    if op == "filtration":  # z[x > 1] = 0
        zero = xg.scalar(0, "int32") if dt == "int32" else xg.scalar(0.0)
        call = Call(L.xtg_filter_assign, [zero, cond], 0, z)
        return {"in": [x], "calls": [call], "out": [z]}
    if op == "masked":  # masked_view(z, m) = x
        m = torch.rand((n,), generator=g, device="cuda") < 0.5
        call = Call(L.xtg_masked_assign, [_arr(x), _arr(m)], 0, z)
        return {"in": [x, m], "calls": [call], "out": [z]}
    idx = torch.randint(0, n, (max(1, n // 8), 1), generator=g, device="cuda")
    out = _empty((idx.shape[0],), dt)
    return {"in": [x, idx], "calls": [Call(L.xtg_gather, [_arr(x)], idx.data_ptr(), idx.shape[0], out)], "out": [out]}


def run(state):
    if "read" in state:
        return state["read"]()
    for c in state["calls"]:
        c()
    return state["out"]


# ---- what it needs, and what it should be ---------------------------------------------


def work(case):
    kind, s = case["kind"], SIZE.get(case.get("dtype", "float32"))
    if kind == "requests":
        got = _requests(case)
        return {"bytes": sum(_request_bytes(*r) for r in got), "flops": sum(2 * math.prod(r[2]) for r in got)}
    if kind == "fused":
        n = case["rows"] * case["cols"]
        return {"bytes": (2 * n + case["cols"] + case["rows"]) * s, "flops": 6 * n}
    if kind == "batch":
        sizes = _instances(case)
        return {"bytes": sum(4 * (2 * r * c + r + c) for r, c in sizes), "flops": sum(3 * r * c for r, c in sizes)}
    if kind == "normalize":
        n = case["rows"] * case["cols"]
        return {"bytes": 2 * n * s, "flops": 6 * n}
    if kind == "moments":
        return {"bytes": case["n"] * s + 32, "flops": 4 * case["n"]}
    if kind == "views":
        n, m = case["n"], case["n"] * (0.25 if case["dtype"] == "int32" else 0.1587)
        b = {"filter": n * s + m * s, "filtration": n * s + m * s, "masked": n * (s + 1) + n * s,
             "gather": n // 8 * (8 + 2 * s)}[case["op"]]
        return {"bytes": int(b), "flops": n}
    n = math.prod(_shape(case))
    if kind == "reduce":
        kept = math.prod(d for i, d in enumerate(_shape(case)) if i not in _axes(case))
        return {"bytes": n * s + kept * SIZE[_result(case["op"], case["dtype"])], "flops": 2 * n}
    if kind == "argmax":
        return {"bytes": n * s + n // _shape(case)[case["axis"]] * 4, "flops": n}
    if kind == "chunked":  # x read, the chunks written and read for the sums
        return {"bytes": 3 * n * s + case["d0"] * case["d1"] * s, "flops": 3 * n}
    return {"bytes": 2 * n * s, "flops": n}  # transpose, cumsum


def exact(case, seed):
    kind, dt = case["kind"], case.get("dtype", "float32")
    if kind == "batch":
        inst, res = _batch_arrays(case, seed)
        want = torch.zeros(res.shape, dtype=torch.float64, device="cuda")
        at = 0
        for A, v, Cm, o in inst:
            want[at:at + o.numel()] = (A.double() * v.double() + Cm.double()).sum(1)
            at += -(-o.numel() // 64) * 64
        return [want]
    g = _gen(seed)
    if kind == "requests":
        return [_request_exact(w, d, _request(w, d, s, g)[0]) for w, d, s in _requests(case)]
    if kind == "fused":
        A = torch.rand((case["rows"], case["cols"]), generator=g, device="cuda", dtype=TORCH[dt]).mul_(2).sub_(1)
        e = A.double() * _values(g, (case["cols"],), dt).double() + torch.exp(-A.double() * A.double())
        return [e, e.sum(1)]
    if kind == "moments":
        x = _lognormal(g, case["n"], dt).double()
        return [x.sum(), x.mean(), x.var(correction=0), x.square_().sum().sqrt()]
    if kind == "views":
        x = _values(g, (case["n"],), dt)
        keep = x > (500 if dt == "int32" else 1.0)
        if case["op"] == "filter":
            got = x[keep].double()
            return [torch.nn.functional.pad(got, (0, x.numel() - got.numel())), None]
        if case["op"] == "filtration":
            return [_values(g, x.shape, dt).double().masked_fill_(keep, 0.0)]
        if case["op"] == "masked":
            z = _values(g, x.shape, dt)
            return [torch.where(torch.rand(x.shape, generator=g, device="cuda") < 0.5, x, z).double()]
        _values(g, x.shape, dt)  # the destination that the writes draw, and a read does not use
        return [x[torch.randint(0, case["n"], (max(1, case["n"] // 8), 1), generator=g, device="cuda")[:, 0]].double()]
    x = _values(g, (case["rows"], case["cols"]) if kind == "normalize" else _shape(case), dt)
    if kind == "transpose":
        return [x.permute([int(c) for c in case["perm"]]).double()]
    if kind == "argmax":
        return None
    if kind == "chunked":
        shape, cs, per, cells = _chunk_grid(case)
        y = x.double() * 2.0 + 1.0
        slab = torch.zeros((per * len(cells),), dtype=torch.float64, device="cuda")
        for i, (at, ext) in enumerate(cells):
            slab[i * per:i * per + math.prod(cs)].view(cs)[tuple(slice(0, e) for e in ext)] = y[at]
        return [slab, y.sum(2)]
    x = x.double()
    if kind == "normalize":
        return [(x - x.mean(1, keepdim=True)) / torch.sqrt(x.var(1, correction=0, keepdim=True) + EPS)]
    if kind == "cumsum":
        return [x.flatten().cumsum(0) if case["axis"] < 0 else x.cumsum(case["axis"])]
    axes = _axes(case)
    return [{"sum": lambda: x.sum(axes), "mean": lambda: x.mean(axes), "amax": lambda: x.amax(axes),
             "variance": lambda: x.var(axes, correction=0), "norm_l2": lambda: x.square().sum(axes).sqrt()}[case["op"]]()]
