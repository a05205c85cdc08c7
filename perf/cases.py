"""The work that users of the k-NN graph builder have it do, as measurable cases.

A case is a dict of plain values.  `listed()` gives the standing ones, `draw(rng)`
one more of the same ranges; `prepare(case, seed)` makes what a program has in
hand before the call (points on the GPU, output buffers, a library context),
`run(state)` makes one call of a public entry point and returns its outputs,
`work(case)` states the bytes and operations that the call cannot do without,
and `exact(case, seed)` gives 64-bit values where the outputs have any.

Entry points: `knn_build_ex` and `knn_build_batch` on device memory and a
program's own stream (the calls return when queued), `knn_build` of the Python
module on host arrays, and `knn_exact_fp64`.
"""
from __future__ import annotations

import ctypes
import importlib.util
import math
import random
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]
PKG_DIR = ROOT / "approximate-cuda-knn_b200"

EUCLIDEAN, TAXICAB, COSINE = 0, 1, 2
PRECISIONS = {"fp32": 0, "bf16": 1, "f16": 2}


def _load_package():
    """Import approximate-cuda-knn_b200/ (not a valid module name) as `acknn`."""
    if "acknn" in sys.modules:
        return sys.modules["acknn"]
    spec = importlib.util.spec_from_file_location(
        "acknn", PKG_DIR / "__init__.py", submodule_search_locations=[str(PKG_DIR)])
    mod = importlib.util.module_from_spec(spec)
    sys.modules["acknn"] = mod
    spec.loader.exec_module(mod)
    return mod


acknn = _load_package()


class _Program:
    """What a program keeps for its lifetime: one library context (device
    scratch reused by every call) and one stream."""

    def __init__(self):
        self.lib = acknn.load_library()
        self.ctx = acknn.Context(0)
        self.stream = torch.cuda.Stream()


_program = None


def _prog() -> _Program:
    global _program
    if _program is None:
        _program = _Program()
    return _program


# ------------------------------------------------------------------ cases --

def listed():
    return [
        # A small set through the Python module, host arrays in and out: the
        # smallest workload of the repository, where launches and latency count.
        dict(name="small_host", kind="host", data="gaussians", n=10_000, d=16, k=10, trees=10, leaf=32,
             props=3, metric=EUCLIDEAN, precision="fp32"),
        # The headline: 1M integer descriptors, BF16 tiles, the cheapest
        # setting that reaches recall 0.95.
        dict(name="headline_bf16", kind="build", data="integer", n=1_000_000, d=128, k=16, trees=8, leaf=2048,
             props=0, metric=EUCLIDEAN, precision="bf16"),
        # The same data at the configuration's literal setting (many trees of
        # small leaves, then propagation), an odd number of points.
        dict(name="literal_bf16", kind="build", data="integer", n=499_979, d=128, k=16, trees=16, leaf=64,
             props=5, metric=EUCLIDEAN, precision="bf16"),
        # Plain FP32 at its own 0.95 setting: programs that want the
        # bit-reproducible graph.
        dict(name="plain_fp32", kind="build", data="integer", n=300_007, d=128, k=16, trees=16, leaf=512,
             props=1, metric=EUCLIDEAN, precision="fp32"),
        # The largest: 10M unit rows stored as FP16, cosine, FP16 tiles.
        dict(name="cosine_f16_10m", kind="build", data="unit_f16", n=10_000_000, d=96, k=10, trees=15, leaf=4096,
             props=0, metric=COSINE, precision="f16"),
        # Plain FP32 cosine, ragged in every size, k above half a warp.
        dict(name="cosine_plain_ragged", kind="build", data="scaled", n=200_003, d=37, k=21, trees=6, leaf=100,
             props=2, metric=COSINE, precision="fp32"),
        # Long sparse rows under L1, the literal setting: propagation dominates.
        dict(name="sparse_l1", kind="build", data="sparse", n=200_000, d=784, k=30, trees=8, leaf=128,
             props=4, metric=TAXICAB, precision="fp32"),
        # The same rows with large leaves, which high recall needs there.
        dict(name="sparse_l1_large_leaf", kind="build", data="sparse", n=250_000, d=784, k=30, trees=4, leaf=32768,
             props=1, metric=TAXICAB, precision="fp32"),
        # Many independent sets in one call, at the mixed path's 0.95 setting ...
        dict(name="batch_bf16", kind="batch", data="gaussians", sets=48, sizes=1, n_lo=1000, n_hi=200_000, k=15,
             trees=3, leaf=4096, props=0, metric=EUCLIDEAN, precision="bf16"),
        # ... and at the literal setting in plain FP32.
        dict(name="batch_plain", kind="batch", data="gaussians", sets=48, sizes=2, n_lo=1000, n_hi=200_000, k=15,
             trees=8, leaf=48, props=3, metric=EUCLIDEAN, precision="fp32"),
        # Learned splits on data where raw coordinates misrepresent the metric:
        # the network's training is most of the call.
        dict(name="learned_cosine", kind="build", data="scaled", n=100_000, d=64, k=10, trees=8, leaf=64,
             props=2, metric=COSINE, precision="fp32", learned=True),
        # The exact FP64 yardstick that recall is measured with.
        dict(name="exact_fp64", kind="exact", data="integer", n=200_000, d=128, k=16, queries=2000,
             metric=EUCLIDEAN),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["build", "build", "build", "build", "build", "batch", "host", "exact"])
    if kind == "exact":
        return dict(kind=kind, data=rng.choice(["integer", "gaussians"]), n=_log_int(rng, 5_000, 200_000),
                    d=_log_int(rng, 8, 200), k=rng.randint(5, 40), queries=rng.randint(100, 2000),
                    metric=rng.choice([EUCLIDEAN, TAXICAB, COSINE]))
    if kind == "batch":
        prec = rng.choice(["fp32", "bf16"])
        return dict(kind=kind, data="gaussians", sets=rng.randint(3, 48), sizes=rng.randint(3, 1 << 20),
                    n_lo=1000, n_hi=_log_int(rng, 5_000, 100_000), k=rng.randint(5, 16), trees=rng.randint(2, 8),
                    leaf=_log_int(rng, 40, 512 if prec == "fp32" else 4096), props=rng.randint(0, 3),
                    metric=rng.choice([EUCLIDEAN, COSINE]), precision=prec)
    if kind == "host":
        return dict(kind=kind, data=rng.choice(["gaussians", "integer"]), n=_log_int(rng, 2_000, 50_000),
                    d=_log_int(rng, 8, 128), k=rng.randint(5, 20), trees=rng.randint(3, 10),
                    leaf=_log_int(rng, 24, 256), props=rng.randint(0, 3),
                    metric=rng.choice([EUCLIDEAN, TAXICAB, COSINE]), precision=rng.choice(["fp32", "bf16"]))
    data = rng.choice(["integer", "integer", "unit_f16", "scaled", "sparse", "gaussians"])
    c = dict(kind=kind, data=data, props=rng.randint(0, 3))
    if data == "sparse":
        c.update(n=_log_int(rng, 5_000, 100_000), d=rng.randint(300, 784), k=rng.randint(10, 30),
                 trees=rng.randint(2, 6), leaf=_log_int(rng, 64, 8192), metric=rng.choice([EUCLIDEAN, TAXICAB]),
                 precision="fp32")
    else:
        prec = rng.choice(["fp32", "bf16", "f16"])
        n_hi, leaf_hi = (300_000, 1024) if prec == "fp32" else (2_000_000, 4096)
        metric = COSINE if data in ("unit_f16", "scaled") else rng.choice([EUCLIDEAN, EUCLIDEAN, COSINE])
        c.update(n=_log_int(rng, 5_000, n_hi), d=_log_int(rng, 16, 256), k=rng.randint(5, 30),
                 trees=rng.randint(3, 12), leaf=_log_int(rng, 48, leaf_hi), metric=metric, precision=prec)
        if data == "scaled" and prec == "fp32" and rng.random() < 0.5:
            c.update(n=_log_int(rng, 20_000, 200_000), learned=True)
    return c


# ------------------------------------------------------------------- data --
# The distributions of the repository's workloads module, drawn on the GPU.

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFFFFFF)
    return g


def _points(data, n, d, seed):
    g = _gen(seed)
    step = 1 << 19

    def mixture(clusters, centres, sigma, out_dtype, finish):
        labels = torch.randint(0, clusters, (n,), generator=g, device="cuda")
        out = torch.empty((n, d), dtype=out_dtype, device="cuda")
        for s in range(0, n, step):
            e = min(n, s + step)
            x = torch.randn((e - s, d), generator=g, device="cuda")
            out[s:e] = finish(x.mul_(sigma).add_(centres[labels[s:e]])).to(out_dtype)
        return out

    if data == "gaussians":  # 16 isotropic clusters, centres U[-10, 10]
        c = torch.rand((16, d), generator=g, device="cuda").mul_(20.0).sub_(10.0)
        return mixture(16, c, 1.0, torch.float32, lambda x: x)
    if data == "integer":  # 256 clusters, integers in [0, 255]
        c = torch.rand((256, d), generator=g, device="cuda").mul_(255.0)
        return mixture(256, c, 20.0, torch.float32, lambda x: x.round_().clamp_(0.0, 255.0))
    if data in ("unit_f16", "scaled"):  # 1000 or 100 clusters of unit rows
        clusters = 1000 if data == "unit_f16" else 100
        c = torch.randn((clusters, d), generator=g, device="cuda")
        x = mixture(clusters, c, 0.3, torch.float16 if data == "unit_f16" else torch.float32,
                    lambda x: x.div_(x.norm(dim=1, keepdim=True)))
        if data == "scaled":  # norms log-uniform in [0.1, 10]
            u = torch.rand((n, 1), generator=g, device="cuda")
            x.mul_(torch.exp(u.mul_(2.0 * math.log(10.0)).sub_(math.log(10.0))))
        return x
    if data == "sparse":  # 10 prototypes' 20 % supports, U(0, 1] there, zero elsewhere
        m = int(round(0.2 * d))
        sup = torch.zeros((10, d), dtype=torch.float32, device="cuda")
        for p in range(10):
            sup[p, torch.randperm(d, generator=g, device="cuda")[:m]] = 1.0
        labels = torch.randint(0, 10, (n,), generator=g, device="cuda")
        out = torch.empty((n, d), device="cuda")
        for s in range(0, n, step):
            e = min(n, s + step)
            out[s:e] = (1.0 - torch.rand((e - s, d), generator=g, device="cuda")) * sup[labels[s:e]]
        return out
    raise ValueError(data)


def _set_shapes(case):
    """(n, d) of a batch's sets: n log-uniform, d of {32, 64, 128, 256}."""
    r = random.Random(case["sizes"])
    return [(_log_int(r, case["n_lo"], case["n_hi"]), r.choice([32, 64, 128, 256])) for _ in range(case["sets"])]


# -------------------------------------------------------------------- run --

def _options(x, case):
    return acknn.default_options(points_on_device=1, outputs_on_device=1, stream=_prog().stream.cuda_stream,
                                 dtype=acknn.F16 if x.dtype == torch.float16 else acknn.F32,
                                 precision=PRECISIONS[case["precision"]],
                                 learned_splits=int(case.get("learned", False)))


def prepare(case, seed):
    p = _prog()
    kind = case["kind"]
    if kind == "batch":
        shapes = _set_shapes(case)
        xs = [_points(case["data"], n, d, seed * 1000 + i) for i, (n, d) in enumerate(shapes)]
        idx = [torch.empty((n, case["k"]), dtype=torch.int32, device="cuda") for n, _ in shapes]
        dist = [torch.empty((n, case["k"]), dtype=torch.float32, device="cuda") for n, _ in shapes]
        table = (acknn.KnnDataset * len(xs))()
        for i, (n, d) in enumerate(shapes):
            table[i].points, table[i].n, table[i].d, table[i].seed = xs[i].data_ptr(), n, d, i
            table[i].out_idx, table[i].out_dist = idx[i].data_ptr(), dist[i].data_ptr()
        st = dict(case=case, xs=xs, idx=idx, dist=dist, table=table, opt=_options(xs[0], case))
    else:
        x = _points(case["data"], case["n"], case["d"], seed)
        if kind == "host":
            st = dict(case=case, x=x.cpu().numpy())
        elif kind == "exact":
            q = torch.randperm(case["n"], generator=_gen(seed + 1), device="cuda")[:case["queries"]].sort().values
            st = dict(case=case, x=x, q=q.cpu().numpy().astype(np.int64),
                      idx=np.empty((case["queries"], case["k"]), dtype=np.int32),
                      dist=np.empty((case["queries"], case["k"]), dtype=np.float64),
                      opt=acknn.default_options(points_on_device=1, stream=p.stream.cuda_stream))
        else:
            st = dict(case=case, x=x, opt=_options(x, case),
                      idx=torch.empty((case["n"], case["k"]), dtype=torch.int32, device="cuda"),
                      dist=torch.empty((case["n"], case["k"]), dtype=torch.float32, device="cuda"))
    # the points were made on torch's current stream; the calls go to the program's
    p.stream.wait_stream(torch.cuda.current_stream())
    return st


def _check(rc):
    if rc:
        raise acknn.KnnError(rc, _prog().lib.knn_last_error().decode())


def run(state):
    c, p = state["case"], _prog()
    kind = c["kind"]
    if kind == "host":
        return acknn.knn_build(state["x"], c["k"], c["trees"], c["leaf"], c["props"], c["metric"], seed=1,
                               precision=PRECISIONS[c["precision"]])
    if kind == "exact":
        _check(p.lib.knn_exact_fp64(p.ctx.handle, state["x"].data_ptr(), c["n"], c["d"], c["k"], c["metric"],
                                    state["q"].ctypes.data, c["queries"], state["idx"].ctypes.data,
                                    state["dist"].ctypes.data, ctypes.byref(state["opt"])))
        return state["idx"], state["dist"]
    if kind == "batch":
        _check(p.lib.knn_build_batch(p.ctx.handle, state["table"], c["sets"], c["k"], c["trees"], c["leaf"],
                                     c["props"], c["metric"], ctypes.byref(state["opt"]), None))
        # one tensor of each kind for all sets, as the program hands them on
        with torch.cuda.stream(p.stream):
            return torch.cat(state["idx"]), torch.cat(state["dist"])
    _check(p.lib.knn_build_ex(p.ctx.handle, state["x"].data_ptr(), c["n"], c["d"], c["k"], c["trees"], c["leaf"],
                              c["props"], c["metric"], 1, state["idx"].data_ptr(), state["dist"].data_ptr(),
                              ctypes.byref(state["opt"]), None))
    return state["idx"], state["dist"]


# ------------------------------------------------------------------- work --

def _build_work(n, d, k, trees, leaf, props, esize):
    depth = 0
    while math.ceil(n / 2 ** depth) > leaf:
        depth += 1
    block = n / 2 ** depth
    # each unordered pair of a leaf once, one projection per (point, tree, level)
    flops = trees * n * (block - 1) / 2 * 2 * d + trees * n * depth * 2 * d
    # points in, graph out; a propagation step reads and writes the lists once
    return n * d * esize + n * k * 8 * (1 + 2 * props), flops


def work(case):
    c = case
    if c["kind"] == "exact":
        return {"bytes": c["n"] * c["d"] * 4 + c["queries"] * c["k"] * 12,
                "flops": 2.0 * c["queries"] * c["n"] * c["d"]}
    if c["kind"] == "batch":
        parts = [_build_work(n, d, c["k"], c["trees"], c["leaf"], c["props"], 4) for n, d in _set_shapes(c)]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    b, f = _build_work(c["n"], c["d"], c["k"], c["trees"], c["leaf"], c["props"],
                       2 if c["data"] == "unit_f16" else 4)
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------ exact --

def exact(case, seed):
    """64-bit distances of the exact search.  A built graph is the outcome of
    seeded random splits; apart from the builder's own splits it has no value
    to compute, so builds give None."""
    c = case
    if c["kind"] != "exact":
        return None
    x = _points(c["data"], c["n"], c["d"], seed).double()
    q = torch.randperm(c["n"], generator=_gen(seed + 1), device="cuda")[:c["queries"]].sort().values
    out = torch.empty((c["queries"], c["k"]), dtype=torch.float64, device="cuda")
    unit = x / x.norm(dim=1, keepdim=True).clamp_min(1e-300) if c["metric"] == COSINE else None
    rows = max(1, (1 << 25) // c["n"])
    for s in range(0, c["queries"], rows):
        qs = q[s:s + rows]
        if c["metric"] == COSINE:
            dm = 1.0 - unit[qs] @ unit.T
        else:
            dm = torch.cdist(x[qs], x, p=2.0 if c["metric"] == EUCLIDEAN else 1.0,
                             compute_mode="donot_use_mm_for_euclid_dist")
        dm[torch.arange(len(qs), device="cuda"), qs] = float("inf")
        out[s:s + rows] = dm.topk(c["k"], dim=1, largest=False).values
    return None, out
