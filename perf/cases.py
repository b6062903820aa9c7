"""Timed cases of the framework's main paths, through its public entry points.

Each case is a dict of plain values:

* ``kind`` "reshape": an array between two decompositions (and back when ``both``);
* ``kind`` "forward": a forward split 3D FFT, returning the spectrum in the plan's B layout;
* ``kind`` "step": reshapes through a chain of decompositions, then a forward and an inverse split FFT on
  the last one, returning the inverse's output;
* ``kind`` "batch": several arrays of one shape, moved from the block to the rotate decomposition in grouped
  launches and transformed forward and back in batched ones (what the request server runs per batch);
* ``kind`` "group": arrays of different small shapes, forward, one launch per pass of all of them.

Arrays are virtual-grid arrays (rank r's buffer at element r * pitch) on ``ranks`` virtual ranks; the
decompositions are spec strings of ``decomp_from_spec``.  Inputs are uniform[-1, 1) values, as in the
benchmark; the spectra's error is what plain float64 FFTs of the same values give in :func:`exact`.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from decomp_mpi_gb300 import api

DEV = "cuda:0"
ELEM = {"i64": torch.int64, "c64": torch.complex64, "c128": torch.complex128}
SIZE = {"i64": 8, "c64": 8, "c128": 16}
ARITH = {"df": api.ARITH_DF, "fp64": api.ARITH_FP64, "fp32": api.ARITH_FP32, "tc16": api.ARITH_TC16}
GROUP_SHAPES = ("32x32x32 48x40x36 64x48x32 40x40x40 24x30x36 60x48x40 72x64x48 80x60x50 96x64x32 30x30x30 "
                "36x48x60 45x40x32 64x64x64 50x40x30 96x96x48 20x24x30")


def _shape(text):
    return tuple(int(v) for v in text.split("x"))


def _blocks(shape, g0, g1):
    return "packed:block(%d,%d)|block(%d,%d)|local(%d)" % (shape[0], g0, shape[1], g1, shape[2])


def _rotated(shape, g0, g1):
    return "packed:rotate(%d,block(%d,%d))|rotate(1,block(%d,%d))|local(%d)" % (
        max(1, shape[0] // 3), shape[0], g0, shape[1], g1, shape[2])


def listed():
    cube = (512, 512, 512)
    chain = ";".join([_blocks(cube, 8, 8),
                      "packed:rotate(1,block(512,8))|rotate(170,block(512,8))|local(512)",
                      "packed:frev(16,32,block(512,8))|frev(32,16,block(512,8))|local(512)"])
    pencils = ";".join(["packed:local(64)|block(64,2)|block(64,2)", "packed:block(64,2)|local(64)|block(64,2)",
                        "packed:block(64,2)|block(64,2)|local(64)"])
    c = (1024, 1024, 1024)
    return [
        # an in-cache redistribution, both ways: the smallest array of the bandwidth sweep
        {"name": "reshape_256_c64", "kind": "reshape", "shape": "256x256x256", "elem": "c64", "ranks": 256,
         "src": _blocks((256, 256, 256), 16, 16), "dst": _rotated((256, 256, 256), 16, 16), "both": True},
        # the sweep's largest: a 4 GiB integer field to the interleaved layout
        {"name": "reshape_large_i64", "kind": "reshape", "shape": "1024x1024x512", "elem": "i64", "ranks": 1024,
         "src": _blocks((1024, 1024, 512), 32, 32),
         "dst": "packed:interleave(block(64,32),16)|interleave(block(64,32),16)|local(512)", "both": False},
        # ragged pencils: uneven blocks on both sides, so every rank has its own strides
        {"name": "reshape_ragged_c128", "kind": "reshape", "shape": "250x333x190", "elem": "c128", "ranks": 35,
         "src": "packed:local(250)|block(333,7)|block(190,5)", "dst": "packed:block(250,7)|block(333,5)|local(190)",
         "both": False},
        # a small solver's step: x to y to z pencils, forward and back (default arithmetic); launches count
        {"name": "pencils_64_c128", "kind": "step", "shape": "64x64x64", "elem": "c128", "ranks": 4, "chain": pencils,
         "arith": "df"},
        # the headline step: reshape chain, forward and inverse in native FP64
        {"name": "step_512_fp64", "kind": "step", "shape": "512x512x512", "elem": "c128", "ranks": 64, "chain": chain,
         "arith": "fp64"},
        # the same array's spectrum in the default complex128 arithmetic
        {"name": "forward_512_df", "kind": "forward", "shape": "512x512x512", "elem": "c128", "ranks": 64,
         "start": chain.split(";")[2], "arith": "df"},
        # the largest: 8 GiB complex64 spectrum
        {"name": "forward_1024_c64", "kind": "forward", "shape": "1024x1024x1024", "elem": "c64", "ranks": 64,
         "start": _blocks(c, 8, 8), "arith": "fp32"},
        # the tensor-core form of the 1024-point lines
        {"name": "forward_1024_tc16", "kind": "forward", "shape": "1024x1024x512", "elem": "c64", "ranks": 64,
         "start": _blocks((1024, 1024, 512), 8, 8), "arith": "tc16"},
        # a server's batch: eight jobs of one 2,3,5-smooth side, forward and back
        {"name": "batch_240_c64", "kind": "batch", "shape": "240x240x240", "elem": "c64", "ranks": 16, "grid": "4x4",
         "count": 8, "arith": "fp32"},
        # sixteen uneven small arrays with one launch per pass
        {"name": "group_small_fp64", "kind": "group", "shapes": GROUP_SHAPES, "elem": "c128", "ranks": 16,
         "grid": "4x4", "arith": "fp64"},
        # one long dimension: the two-stage schedule with its split twiddle
        {"name": "forward_4096_df", "kind": "forward", "shape": "4096x128x128", "elem": "c128", "ranks": 16,
         "start": _blocks((4096, 128, 128), 4, 4), "arith": "df"},
        # ragged transform: lengths without kernels of their own, uneven blocks
        {"name": "forward_ragged_df", "kind": "forward", "shape": "180x150x105", "elem": "c128", "ranks": 28,
         "start": _blocks((180, 150, 105), 7, 4), "arith": "df"},
    ]


def _side(rng, lo, hi):
    """A 2,3,5,7-smooth side of [lo, hi], even over the logarithm; odd ones among them."""
    while True:
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        m = n
        for p in (2, 3, 5, 7):
            while m % p == 0:
                m //= p
        if m == 1:
            return n


def _grid_of(rng, n, most):
    """A processor count for one dimension that leaves no rank empty."""
    return rng.choice([g for g in range(1, most + 1) if -(-n // -(-n // g)) == g])


def _decomp(rng, shape, g0, g1):
    a, b, c = shape
    how = rng.choice(["block", "rotate", "frev", "interleave"])
    if how == "block":
        return _blocks(shape, g0, g1)
    if how == "rotate":
        return _rotated(shape, g0, g1)
    if how == "frev":
        def dim(n, g):
            f = rng.choice([d for d in range(1, n + 1) if n % d == 0])
            return "frev(%d,%d,block(%d,%d))" % (f, n // f, n, g)
    else:
        def dim(n, g):
            f = rng.choice([d for d in range(1, n + 1) if n % d == 0 and d >= g and -(-d // -(-d // g)) == g] or [n])
            return "interleave(block(%d,%d),%d)" % (f, g, n // f)
    return "packed:%s|%s|local(%d)" % (dim(a, g0), dim(b, g1), c)


def draw(rng: random.Random):
    kind = rng.choice(["reshape", "reshape", "forward", "forward", "forward", "step", "batch"])
    if kind == "reshape":
        elem = rng.choice(["i64", "c64", "c128"])
        while True:
            shape = tuple(int(round(math.exp(rng.uniform(math.log(24), math.log(1024))))) for _ in range(3))
            if 1 << 16 <= math.prod(shape) <= 1 << 28:
                break
        g0, g1 = (_grid_of(rng, n, 8) for n in shape[:2])
        return {"kind": "reshape", "shape": "%dx%dx%d" % shape, "elem": elem, "ranks": g0 * g1,
                "src": _blocks(shape, g0, g1), "dst": _decomp(rng, shape, g0, g1), "both": rng.random() < 0.5}
    elem = rng.choice(["c64", "c128"])
    arith = rng.choice(["df", "fp64"]) if elem == "c128" else "fp32"
    while True:
        if rng.random() < 0.3:
            side = _side(rng, 24, 512)
            shape = (side, side, side)
        else:
            shape = tuple(_side(rng, 24, 1024) for _ in range(3))
        if 1 << 14 <= math.prod(shape) <= (1 << 26 if kind == "forward" else 1 << 25):
            break
    if elem == "c64" and 1024 in shape and rng.random() < 0.5:
        arith = "tc16"
    g0, g1 = (_grid_of(rng, n, 6) for n in shape[:2])
    base = {"kind": kind, "shape": "%dx%dx%d" % shape, "elem": elem, "ranks": g0 * g1, "arith": arith}
    if kind == "forward":
        return dict(base, start=_decomp(rng, shape, g0, g1))
    if kind == "step":
        return dict(base, chain=_blocks(shape, g0, g1) + ";" + _decomp(rng, shape, g0, g1))
    most = max(1, min(16, (1 << 25) // math.prod(shape)))
    return dict(base, grid="%dx%d" % (g0, g1), count=rng.randint(min(2, most), most))


# ---------------------------------------------------------------- what a user's program holds

def _uniform(n, elem, gen):
    if elem == "i64":
        return torch.randint(-(1 << 62), 1 << 62, (n,), dtype=torch.int64, device=DEV, generator=gen)
    t = torch.empty(n, dtype=ELEM[elem], device=DEV)
    torch.view_as_real(t).uniform_(-1, 1, generator=gen)
    return t


def _generator(seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    return gen


def _split_plan(start, dat, P, case):
    """A plan on `dat` with the workspace it asks for."""
    dtype = api.C128 if case["elem"] == "c128" else api.C64
    probe = api.SplitPlan(start, 1 << 20, 1 << 40, 1 << 21, dtype=dtype)
    ext = probe.extent64
    probe.free()
    work = torch.zeros(P * 2 * ext, dtype=ELEM[case["elem"]], device=DEV)
    plan = api.SplitPlan(start, dat.data_ptr(), 2 * ext, work.data_ptr(), dtype=dtype, arith=ARITH[case["arith"]])
    return plan, work, ext


def prepare(case, seed):
    P, kind, elem = case["ranks"], case["kind"], case["elem"]
    comm = api.Comm(P)
    gen = _generator(seed)
    s = {"case": case, "comm": comm}
    if kind == "reshape":
        a, b = (api.decomp_from_spec(comm, case[k]) for k in ("src", "dst"))
        s["plan"] = api.ReshapePlan(comm, SIZE[elem], a, b)
        s["src"] = _uniform(P * s["plan"].src_pitch, elem, gen)
        s["dst"] = torch.zeros(P * s["plan"].dest_pitch, dtype=ELEM[elem], device=DEV)
        if case["both"]:
            s["back"] = api.ReshapePlan(comm, SIZE[elem], b, a)
            s["again"] = torch.zeros_like(s["src"])
        s["decomps"] = (a, b)
    elif kind == "forward":
        start = api.decomp_from_spec(comm, case["start"])
        s["dat"] = _uniform(P * start.extent(), elem, gen)
        s["plan"], s["work"], s["ext"] = _split_plan(start, s["dat"], P, case)
        s["decomps"] = (start,)
    elif kind == "step":
        decomps = [api.decomp_from_spec(comm, t) for t in case["chain"].split(";")]
        s["moves"] = [api.ReshapePlan(comm, SIZE[elem], a, b) for a, b in zip(decomps, decomps[1:])]
        s["arrays"] = [_uniform(P * decomps[0].extent(), elem, gen)]
        s["arrays"] += [torch.zeros(P * d.extent(), dtype=ELEM[elem], device=DEV) for d in decomps[1:]]
        s["plan"], s["work"], s["ext"] = _split_plan(decomps[-1], s["arrays"][-1], P, case)
        s["decomps"] = decomps
    elif kind == "batch":
        shape, (g0, g1) = _shape(case["shape"]), _shape(case["grid"])
        block, rot = (api.decomp_from_spec(comm, f(shape, g0, g1)) for f in (_blocks, _rotated))
        s["inputs"] = [_uniform(P * block.extent(), elem, gen) for _ in range(case["count"])]
        s["dats"] = [torch.zeros(P * rot.extent(), dtype=ELEM[elem], device=DEV) for _ in s["inputs"]]
        s["move"] = api.ReshapePlan(comm, SIZE[elem], block, rot)
        s["plan"], work, ext = _split_plan(rot, s["dats"][0], P, case)
        s["works"] = [work] + [torch.zeros_like(work) for _ in s["inputs"][1:]]
        s["scales"] = torch.zeros(case["count"], 64, dtype=torch.int32, device=DEV)
        s["decomps"] = (block, rot)
    else:
        g0, g1 = _shape(case["grid"])
        s["starts"], s["dats"], s["plans"], s["works"], s["exts"] = [], [], [], [], []
        for text in case["shapes"].split():
            start = api.decomp_from_spec(comm, _blocks(_shape(text), g0, g1))
            dat = _uniform(P * start.extent(), elem, gen)
            plan, work, ext = _split_plan(start, dat, P, case)
            plan.set_radix(api.RADIX_PLAN8)
            for k, v in zip(("starts", "dats", "plans", "works", "exts"), (start, dat, plan, work, ext)):
                s[k].append(v)
    return s


def run(s):
    case = s["case"]
    kind, P = case["kind"], case["ranks"]
    sh = torch.cuda.current_stream().cuda_stream
    if kind == "reshape":
        s["plan"].run(s["src"].data_ptr(), s["dst"].data_ptr(), sh)
        if not case["both"]:
            return s["dst"]
        s["back"].run(s["dst"].data_ptr(), s["again"].data_ptr(), sh)
        return [s["dst"], s["again"]]
    if kind == "forward":
        s["plan"].run(api.FFTW_FORWARD, sh)
        return s["work"].view(P, -1)[:, :s["ext"]]
    if kind == "step":
        for move, a, b in zip(s["moves"], s["arrays"], s["arrays"][1:]):
            move.run(a.data_ptr(), b.data_ptr(), sh)
        s["plan"].run(api.FFTW_FORWARD, sh)
        s["plan"].run(api.FFTW_BACKWARD, sh)
        return s["arrays"][-1]
    if kind == "batch":
        n = case["count"]
        dats, works = [t.data_ptr() for t in s["dats"]], [t.data_ptr() for t in s["works"]]
        scales = [t.data_ptr() for t in s["scales"]]
        api.reshape_group([s["move"]] * n, [t.data_ptr() for t in s["inputs"]], dats, sh)
        s["plan"].run_batch(api.FFTW_FORWARD, dats, works, scales, sh)
        s["plan"].run_batch(api.FFTW_BACKWARD, dats, works, scales, sh)
        return list(s["dats"])
    api.split_run_group(s["plans"], api.FFTW_FORWARD, sh)
    return [w.view(P, -1)[:, :e] for w, e in zip(s["works"], s["exts"])]


def work(case):
    """Each input read once and each output written once (the passes between them could stay on the chip only
    for small arrays, but they are no part of what the call is asked for); flops by 5 N log2 N a transform."""
    size = SIZE[case["elem"]]
    if case["kind"] == "group":
        points = [math.prod(_shape(t)) for t in case["shapes"].split()]
        return {"bytes": 2 * size * sum(points), "flops": sum(5 * n * math.log2(n) for n in points)}
    n = math.prod(_shape(case["shape"]))
    flops = 5 * n * math.log2(n)
    if case["kind"] == "reshape":
        return {"bytes": (4 if case["both"] else 2) * n * size, "flops": 0}
    if case["kind"] == "batch":
        return {"bytes": case["count"] * 2 * n * size, "flops": case["count"] * 2 * flops}
    return {"bytes": 2 * n * size, "flops": flops * (2 if case["kind"] == "step" else 1)}


# ---------------------------------------------------------------- the outputs in plain float64

def _local(n):
    return np.zeros(n, np.int64), np.arange(n), 1


def _block(n, procs, factor=1):
    size = factor * -(-(n // factor) // procs)
    x = np.arange(n)
    return x // size, x % size, procs


def _rotate(r, nested):
    x = (np.arange(len(nested[0])) + r) % len(nested[0])
    return nested[0][x], nested[1][x], nested[2]


def _frev(a, b, nested):
    x = np.arange(a * b)
    x = x // a + b * (x % a)
    return nested[0][x], nested[1][x], nested[2]


def _interleave(nested, b):
    a = len(nested[0])
    x = np.arange(a * b)
    return nested[0][x % a], x // a + b * nested[1][x % a], nested[2]


def _axes(spec):
    names = {"block": _block, "local": _local, "rotate": _rotate, "frev": _frev, "interleave": _interleave}
    return [eval(t, {"__builtins__": {}}, names) for t in spec[len("packed:"):].split("|")]


def _layout(axes):
    """(rank, offset) of every element of a packed decomposition as tensors over the array, and its extent."""
    procs = [a[2] for a in axes]
    held = [np.array([int(a[1][a[0] == p].max()) + 1 if (a[0] == p).any() else 0 for p in range(a[2])]) for a in axes]
    rank, offset = None, None
    strides = np.ones(procs, np.int64)  # of the dimension at hand, by the ranks' positions
    extent = np.ones(procs, np.int64)
    t = [torch.from_numpy(np.ascontiguousarray(a[0])).to(DEV) for a in axes]
    rank_stride = 1
    for i in reversed(range(len(axes))):
        shape = [-1 if k == i else 1 for k in range(len(axes))]
        part = t[i].view(shape)
        rank = part * rank_stride if rank is None else rank + part * rank_stride
        rank_stride *= procs[i]
    flat = []
    for i in reversed(range(len(axes))):
        shape = [-1 if k == i else 1 for k in range(len(axes))]
        flat.append((i, torch.from_numpy(strides.reshape(-1).copy()).to(DEV)))
        n = held[i].reshape(shape)
        extent = extent + strides * (n - 1)
        strides = strides * n
    full = np.ones(procs, bool)
    for i in range(len(axes)):
        full = full & (held[i] > 0).reshape([-1 if k == i else 1 for k in range(len(axes))])
    for i, st in flat:
        shape = [-1 if k == i else 1 for k in range(len(axes))]
        part = torch.from_numpy(np.ascontiguousarray(axes[i][1])).to(DEV).view(shape)
        part = part * (st[0] if bool((st == st[0]).all()) else st[rank])
        offset = part if offset is None else offset + part
    return rank, offset, int(extent[full].max())


def _processor_grid(ranks, tasks):
    """The grid the plan builders choose: least load, then the evenest per-rank task counts."""
    best = {"grid": None, "load": math.prod(tasks), "ratio": 10000.0}

    def walk(dim, grid, procs, load, lo, hi):
        for g in range(1, min(ranks, tasks[dim]) + 1):
            if procs * g > ranks:
                break
            low, high = min(lo, tasks[dim] // g), max(hi, -(-tasks[dim] // g))
            new = load * -(-tasks[dim] // g)
            if dim + 1 < len(tasks):
                walk(dim + 1, grid + [g], procs * g, new, low, high)
            elif new < best["load"] or (new == best["load"] and high / low < best["ratio"]):
                best.update(grid=grid + [g], load=new, ratio=high / low)

    walk(0, [], 1, 1, max(tasks), 0)
    return best["grid"]


def _factors(n):
    a = max(q for q in range(1, n + 1) if n % q == 0 and (q <= n // q) and q < max(n, 2))
    return a, n // a


def _spectrum(case, shape, start, x):
    """The forward transform of the start layout's values x in the plan's workspace (every rank's first extent)."""
    P = case["ranks"]
    rank, offset, pitch = _layout(_axes(start))
    f = x.view(-1)[rank * pitch + offset].to(torch.complex128)
    del rank, offset
    for d in reversed(range(3)):
        f = torch.fft.fft(f, dim=d)
    A, B = zip(*(_factors(n) for n in shape))
    ga, gb = _processor_grid(P, A), _processor_grid(P, B)
    _, _, ext = _layout([_interleave(_block(a, g), b) for a, b, g in zip(A, B, ga)])
    rank, offset, ext_b = _layout([_block(n, g, a) for n, a, g in zip(shape, A, gb)])
    ext = max(ext, ext_b)
    out = torch.zeros(P * ext, dtype=torch.complex128, device=DEV)
    for d in range(3):  # slot s of dimension d holds frequency s // A + B * (s % A)
        s = torch.arange(shape[d], device=DEV)
        f = f.index_select(d, s // A[d] + B[d] * (s % A[d]))
    out[(rank * ext + offset).reshape(-1)] = f.reshape(-1)
    return out.view(P, ext)


def exact(case, seed):
    kind, elem, P = case["kind"], case["elem"], case["ranks"]
    if kind == "reshape":
        return None  # values moved, not computed
    gen = _generator(seed)
    if kind == "forward":
        shape = _shape(case["shape"])
        pitch = _layout(_axes(case["start"]))[2]
        return _spectrum(case, shape, case["start"], _uniform(P * pitch, elem, gen))
    if kind == "group":
        g0, g1 = _shape(case["grid"])
        out = []
        for text in case["shapes"].split():
            start = _blocks(_shape(text), g0, g1)
            pitch = _layout(_axes(start))[2]
            out.append(_spectrum(case, _shape(text), start, _uniform(P * pitch, elem, gen)))
        return out
    # forward and inverse: N times the moved input
    shape = _shape(case["shape"])
    if kind == "step":
        specs = case["chain"].split(";")
        first, last, count = specs[0], specs[-1], 1
    else:
        g0, g1 = _shape(case["grid"])
        first, last, count = _blocks(shape, g0, g1), _rotated(shape, g0, g1), case["count"]
    rank, offset, pitch = _layout(_axes(first))
    src = (rank * pitch + offset).reshape(-1)
    rank, offset, pitch2 = _layout(_axes(last))
    dst = (rank * pitch2 + offset).reshape(-1)
    out = []
    for _ in range(count):
        x = _uniform(P * pitch, elem, gen)
        y = torch.zeros(P * pitch2, dtype=torch.complex128, device=DEV)
        y[dst] = x[src].to(torch.complex128) * math.prod(shape)
        out.append(y)
    return out[0] if kind == "step" else out
