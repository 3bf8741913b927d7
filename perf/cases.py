"""The calls whose speed is watched: what programs written on this package
spend their time in, each through a public entry point, with its inputs, its
compulsory work and its result in 64 bits.

Sizes and distributions are those of the benchmark's configurations
(`bench.py`, `finchgb/workloads.py`) and of the tests around them: matrices
with uniform (Poisson) and with power-law (Zipf 1.5) row lengths, random
graphs, and the 5-point Poisson matrix.  Inputs are made on the GPU from the
seed.
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]
for _p in (ROOT, ROOT / "finch.jl_gb300"):
    if str(_p) not in sys.path:
        sys.path.insert(0, str(_p))

import finchgb as fg  # noqa: E402
from finchgb import _lib as L  # noqa: E402
from finchgb import cg, device, examples, plan  # noqa: E402
from finchgb.workloads import SparseBuffers  # noqa: E402

DTYPES = {"f64": torch.float64, "f32": torch.float32, "bf16": torch.bfloat16, "i32": torch.int32, "i64": torch.int64}
SEMIRINGS = {"plus_times": L.PLUS_TIMES, "min_plus": L.MIN_PLUS, "max_plus": L.MAX_PLUS}


def _size(t):
    return {"f64": 8, "f32": 4, "bf16": 2, "i32": 4, "i64": 8}[t]


def listed():
    return [
        # one small product of a CSC matrix, the benchmark's first
        # configuration: launches and latency are all of it
        {"name": "spmv_small", "op": "spmv", "m": 10_000, "n": 10_000, "mean": 10.0, "dist": "uniform", "val": "f64",
         "vec": "f64", "orient": "csc", "semiring": "plus_times", "accumulate": False},
        # a product with a large skewed matrix (web or social graph), as an
        # iterative method calls it with no plan
        {"name": "spmv_zipf", "op": "spmv", "m": 1_000_000, "n": 1_000_000, "mean": 16.0, "dist": "zipf", "val": "f64",
         "vec": "f64", "orient": "csr", "semiring": "plus_times", "accumulate": False},
        # one relaxation round of single-source shortest paths on the 4M-node
        # graph: whole numbers, accumulating into the distances
        {"name": "minplus_graph", "op": "spmv", "m": 4_000_000, "n": 4_000_000, "mean": 8.0, "dist": "uniform",
         "val": "i32", "vec": "i32", "orient": "csr", "semiring": "min_plus", "accumulate": True},
        # the PageRank example, whole: degrees, transition matrix, 20 steps
        {"name": "pagerank", "op": "pagerank", "m": 1_000_000, "mean": 7.0, "steps": 20},
        # the headline product, planned once and replayed, as a training or
        # solver loop keeps it
        {"name": "spmm_plan", "op": "spmm", "m": 1_000_000, "n": 1_000_000, "mean": 16.0, "dist": "zipf", "k": 128,
         "val": "f32", "vec": "f32", "route": "plan"},
        # a feature-matrix product of ordinary size, ragged shape, written as
        # a lazy expression and run once per matrix (sampled subgraphs)
        {"name": "spmm_lazy", "op": "spmm", "m": 150_011, "n": 120_007, "mean": 12.0, "dist": "zipf", "k": 64,
         "val": "f32", "vec": "f32", "route": "lazy"},
        # a block of right-hand sides in FP64 whose width fits no vector
        {"name": "spmm_odd_f64", "op": "spmm", "m": 200_003, "n": 200_003, "mean": 10.0, "dist": "uniform", "k": 33,
         "val": "f64", "vec": "f64", "route": "call"},
        # sampled dense-dense product on the large skewed pattern: attention
        # scores or the gradient of a sparse weight
        {"name": "sddmm_zipf", "op": "sddmm", "m": 1_000_000, "n": 1_000_000, "mean": 16.0, "dist": "zipf", "k": 64,
         "val": "f32"},
        # the sum of two graphs' weights: a sparse result
        {"name": "ewise_add", "op": "ewise", "m": 2_000_000, "n": 2_000_000, "mean": 8.0, "dist": "uniform",
         "val": "f64", "fn": "add", "orient": "csr"},
        # row sums of an elementwise product of two skewed matrices
        {"name": "ewise_reduce", "op": "ewise_reduce", "m": 500_009, "n": 500_009, "mean": 16.0, "dist": "zipf",
         "val": "f32", "dims": 2, "orient": "csr"},
        # the square of the 5-point matrix, as a multigrid set-up forms it
        {"name": "spgemm_poisson", "op": "spgemm", "grid": 2048, "m": 0, "mean": 0.0, "val": "f64"},
        # the mixed-precision solve of the 2048 x 2048 Poisson problem, whole
        {"name": "cg_poisson", "op": "cg", "grid": 2048, "precision": "bf16", "accumulate": "spmv_pair",
         "rtol": 1e-10},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["spmv", "spmv", "spmv", "spmm", "spmm", "spmm", "sddmm", "ewise", "ewise_reduce", "spgemm",
                     "pagerank", "cg"])
    mean = round(math.exp(rng.uniform(math.log(2.0), math.log(24.0))), 2)
    dist = rng.choice(["uniform", "zipf"])
    if op == "spmv":
        m, n = _log(rng, 1_000, 4_000_000), _log(rng, 1_000, 4_000_000)
        mean = min(mean, n / 8, 32e6 / m)
        semiring = rng.choice(["plus_times", "plus_times", "min_plus", "max_plus"])
        val, vec = rng.choice([("f64", "f64"), ("f32", "f32"), ("i32", "i32"), ("i64", "i64")]
                              + ([("bf16", "f32")] if semiring == "plus_times" else []))
        return {"op": op, "m": m, "n": n, "mean": mean, "dist": dist, "val": val, "vec": vec,
                "orient": rng.choice(["csr", "csr", "csc"]), "semiring": semiring, "accumulate": rng.random() < 0.3}
    if op == "spmm":
        m, n = _log(rng, 1_000, 1_000_000), _log(rng, 1_000, 1_000_000)
        mean = min(mean, n / 8, 16e6 / m)
        vec = rng.choice(["f32", "f32", "f64"])
        val = rng.choice(["f32", "f32", "bf16"]) if vec == "f32" else "f64"
        k = rng.choice([rng.randint(1, 128), 4 * rng.randint(1, 32), rng.choice([8, 16, 32, 64, 128])])
        return {"op": op, "m": m, "n": n, "mean": mean, "dist": dist, "k": k, "vec": vec, "val": val,
                "route": rng.choice(["call", "plan"] if val == "bf16" else ["call", "call", "lazy", "plan"])}
    if op == "sddmm":
        m, n = _log(rng, 1_000, 1_000_000), _log(rng, 1_000, 1_000_000)
        return {"op": op, "m": m, "n": n, "mean": min(mean, n / 8, 16e6 / m), "dist": dist,
                "k": rng.choice([rng.randint(1, 128), 4 * rng.randint(1, 32)]), "val": rng.choice(["f32", "f32", "f64"])}
    if op in ("ewise", "ewise_reduce"):
        m, n = _log(rng, 1_000, 2_000_000), _log(rng, 1_000, 2_000_000)
        c = {"op": op, "m": m, "n": n, "mean": min(mean, n / 8, 16e6 / m), "dist": dist,
             "orient": rng.choice(["csr", "csc"])}
        if op == "ewise":
            return {**c, "val": rng.choice(["f64", "f32", "i32", "i64"]), "fn": rng.choice(["add", "mul"])}
        return {**c, "val": rng.choice(["f64", "f32"]), "dims": rng.choice([0, 1, 2])}
    if op == "spgemm":
        if rng.random() < 0.5:
            return {"op": op, "grid": _log(rng, 64, 2048), "m": 0, "mean": 0.0, "val": rng.choice(["f64", "f32"])}
        return {"op": op, "grid": 0, "m": _log(rng, 1_000, 1_000_000), "mean": round(rng.uniform(2.0, 8.0), 2),
                "val": rng.choice(["f64", "f32"])}
    if op == "pagerank":
        return {"op": op, "m": _log(rng, 10_000, 2_000_000), "mean": round(rng.uniform(3.0, 12.0), 2),
                "steps": rng.choice([10, 20, 30])}
    precision, accumulate = rng.choice([("f64", "f64"), ("f32", "spmv_pair"), ("bf16", "spmv_pair"), ("f32", "f64")])
    return {"op": "cg", "grid": _log(rng, 64, 1024), "precision": precision, "accumulate": accumulate,
            "rtol": rng.choice([1e-8, 1e-10])}


# ---------------------------------------------------------------- inputs


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _lengths(c, m, n, mean, seed, g):
    """Stored entries per fiber: Poisson(mean), or Zipf(1.5) capped at 50,000
    and scaled to the mean by stochastic rounding."""
    if c.get("dist", "uniform") == "uniform":
        return torch.poisson(torch.full((m,), float(mean), device="cuda"), generator=g).long().clamp_(max=n)
    raw = np.minimum(np.random.default_rng(seed).zipf(1.5, size=m), 50_000).astype(np.float64)
    want = torch.from_numpy(raw * (m * mean / raw.sum())).cuda()
    low = want.floor()
    up = torch.rand(m, device="cuda", generator=g, dtype=torch.float64) < want - low
    return (low.long() + up.long()).clamp_(max=n)


def _values(kind, n, g):
    if kind in ("i32", "i64"):
        return torch.randint(1, 1001, (n,), device="cuda", generator=g, dtype=DTYPES[kind])
    if kind == "f64":
        return torch.rand(n, device="cuda", generator=g, dtype=torch.float64)
    return torch.randn(n, device="cuda", generator=g).to(DTYPES[kind])


def _from_keys(key, m, n, val, orient):
    """Finch's level buffers (counted from 1, 32-bit in HBM) of the sorted
    keys fiber * n + coordinate."""
    fib = torch.div(key, n, rounding_mode="floor")
    ptr = torch.ones(m + 1, dtype=torch.int64, device="cuda")
    ptr[1:] += torch.cumsum(torch.bincount(fib, minlength=m), 0)
    idx = (key - fib * n + 1).to(torch.int32)
    shape = (m, n) if orient == "csr" else (n, m)
    return device.DeviceSparse(*shape, ptr.to(torch.int32), idx, val, orient, 1)


def _distinct(fib, ne, nf, want, g, taken=None):
    """`want` distinct sorted keys fiber * ne + coordinate with uniform
    coordinates in the fibers `fib`, none of them in the sorted `taken`."""
    key = fib * ne + torch.randint(0, ne, (fib.numel(),), device="cuda", generator=g)
    while True:
        key = torch.unique(key)
        if taken is not None:
            at = torch.searchsorted(taken, key).clamp_(max=taken.numel() - 1)
            key = key[taken[at] != key]
        short = want - key.numel()
        if short <= 0:
            break
        key = torch.cat([key, torch.randint(0, nf * ne, (short,), device="cuda", generator=g)])
    return _some(key, want, g)


def _some(key, want, g):
    """`want` of the sorted keys, chosen at random, still sorted."""
    return key[torch.randperm(key.numel(), device="cuda", generator=g)[:want].sort().values]


def _matrix(c, seed, val, orient="csr"):
    """A random matrix of `m` rows and `n` columns with m * mean stored
    entries: distinct uniform coordinates in every fiber of the compressed
    direction."""
    g = _gen(seed)
    nf, ne = (c["m"], c["n"]) if orient == "csr" else (c["n"], c["m"])
    want = int(c["m"] * c["mean"])
    lengths = _lengths(c, nf, ne, c["mean"] * c["m"] / nf, seed, g)
    fib = torch.repeat_interleave(torch.arange(nf, device="cuda"), lengths)
    key = _distinct(fib, ne, nf, want, g)
    return _from_keys(key, nf, ne, None if val is None else _values(val, want, g), orient)


def _poisson2d(N, val):
    n = N * N
    r = torch.arange(n, device="cuda")
    i, j = r // N, r % N
    cols, ok, vals = [], [], []
    for di, dj, v in ((-1, 0, -1.0), (0, -1, -1.0), (0, 0, 4.0), (0, 1, -1.0), (1, 0, -1.0)):
        ok.append((i + di >= 0) & (i + di < N) & (j + dj >= 0) & (j + dj < N))
        cols.append(r + di * N + dj)
        vals.append(torch.full((n,), v, dtype=DTYPES[val], device="cuda"))
    ok = torch.stack(ok, 1)
    ptr = torch.ones(n + 1, dtype=torch.int64, device="cuda")
    ptr[1:] += torch.cumsum(ok.sum(1), 0)
    idx = (torch.stack(cols, 1)[ok] + 1).to(torch.int32)
    return device.DeviceSparse(n, n, ptr.to(torch.int32), idx, torch.stack(vals, 1)[ok], "csr", 1)


def _host(A, orient=None):
    """The matrix as Finch's own host buffers (Int64, counted from 1)."""
    ptr, idx, val = A.to_host()
    return SparseBuffers(A.nrows, A.ncols, ptr, idx, val, orient or A.orient)


def prepare(case, seed):
    c, op = case, case["op"]
    g = _gen(seed + 7919)
    if op == "spmv":
        A = _matrix(c, seed, c["val"], c["orient"])
        s = {"case": c, "A": A, "x": _values(c["vec"], c["n"], g)}
        if c["semiring"] != "plus_times" and c["vec"] in ("i32", "i64"):
            # distances: some nodes reached, the others at a large number that a weight does not wrap
            far = torch.rand(c["n"], device="cuda", generator=g) < 0.3
            s["x"][far] = (1 << 30) if c["semiring"] == "min_plus" else -(1 << 30)
        if c["accumulate"]:
            s["y0"] = _values(c["vec"], c["m"], g)
        return s
    if op == "spmm":
        A = _matrix(c, seed, c["val"])
        B = _values(c["vec"], c["n"] * c["k"], g).reshape(c["n"], c["k"])
        s = {"case": c, "A": A, "B": B}
        if c["route"] == "plan":
            s["C"] = torch.empty((c["m"], c["k"]), dtype=B.dtype, device="cuda")
            torch.cuda.synchronize()  # a plan times its candidates on a stream of its own
            s["plan"] = plan.Plan.spmm(A, B, s["C"])
        elif c["route"] == "lazy":
            zero = np.float32(0) if c["vec"] == "f32" else 0.0
            # a CSR matrix is the swizzle of its transpose's CSC
            body = fg.Tensor.from_buffers(fg.Dense(fg.SparseList(fg.Element(zero))), _host(A.T()))
            s["tA"] = fg.swizzle(fg.transfer(fg.gpu(), body), 2, 1)
            s["tB"] = fg.transfer(fg.gpu(), fg.Tensor(fg.Dense(fg.Dense(fg.Element(zero))), B.cpu().numpy()))
        return s
    if op == "sddmm":
        A = _matrix(c, seed, c["val"])
        x, y = (torch.randn((r, c["k"]), device="cuda", generator=g, dtype=DTYPES[c["val"]]) for r in (c["m"], c["n"]))
        return {"case": c, "A": A, "X": x, "Y": y}
    if op in ("ewise", "ewise_reduce"):
        kind = "f64" if op == "ewise_reduce" else c["val"]  # weights that are summed: U[0, 1)
        A = _matrix(c, seed, kind, c["orient"])
        # the second matrix has half of the first one's places and as many
        # others in the same fibers, as two versions of one graph do
        key, nf, ne = _keyed(A)
        kept = _some(key, key.numel() // 2, g)
        moved = key[torch.randperm(key.numel(), device="cuda", generator=g)[:key.numel() - kept.numel()]]
        new = _distinct(torch.div(moved, ne, rounding_mode="floor"), ne, nf, moved.numel(), g, taken=key)
        key = torch.cat([kept, new]).sort().values
        B = _from_keys(key, nf, ne, _values(kind, key.numel(), g), c["orient"])
        A.val, B.val = A.val.to(DTYPES[c["val"]]), B.val.to(DTYPES[c["val"]])
        return {"case": c, "A": A, "B": B}
    if op == "spgemm":
        if c["grid"]:
            A = _poisson2d(c["grid"], c["val"])
            # coefficients that vary from cell to cell
            A = device.DeviceSparse(A.nrows, A.ncols, A.ptr, A.idx, A.val * (0.5 + _values(c["val"], A.nnz, g).abs()),
                                    "csr", 1)
            return {"case": c, "A": A, "B": A}
        # two fixed patterns, new coefficients
        sq = {"m": c["m"], "n": c["m"], "mean": c["mean"]}
        A, B = (_matrix(sq, k, None) for k in (1, 2))
        A.val, B.val = (_values(c["val"], t.nnz, g) for t in (A, B))
        return {"case": c, "A": A, "B": B}
    if op == "pagerank":
        # column j holds j's out-edges: 1 + Poisson(mean) of them, distinct targets
        m = c["m"]
        deg = 1 + torch.poisson(torch.full((m,), c["mean"], device="cuda"), generator=g).long()
        fib = torch.repeat_interleave(torch.arange(m, device="cuda"), deg)
        key = torch.unique(fib * m + torch.randint(0, m, (fib.numel(),), device="cuda", generator=g))
        E = _from_keys(key, m, m, None, "csc")
        t = fg.Tensor.from_buffers(fg.Dense(fg.SparseList(fg.Pattern())), _host(E))
        return {"case": c, "E": E, "edges": fg.transfer(fg.gpu(), t)}
    A = _poisson2d(c["grid"], "f64")
    low = None if c["precision"] == "f64" else cg.low_precision_copy(A, c["precision"])
    b = 2 * torch.rand(A.nrows, device="cuda", generator=g, dtype=torch.float64) - 1
    return {"case": c, "A": A, "low": low, "b": b}


# ---------------------------------------------------------------- one pass


def run(state):
    s, c = state, state["case"]
    op = c["op"]
    if op == "spmv":
        if c["accumulate"]:
            y = s["y0"].clone()
            return fg.spmv(s["A"], s["x"], y, semiring=SEMIRINGS[c["semiring"]], flags=L.ACCUMULATE)
        return fg.spmv(s["A"], s["x"], semiring=SEMIRINGS[c["semiring"]])
    if op == "spmm":
        if c["route"] == "plan":
            s["plan"].execute()
            return s["C"]
        if c["route"] == "lazy":
            return fg.compute(fg.lazy(s["tA"]) @ fg.lazy(s["tB"])).ddata
        return fg.spmm(s["A"], s["B"])
    if op == "sddmm":
        return fg.sddmm(s["A"], s["X"], s["Y"])
    if op == "ewise":
        C = fg.ewise(L.EW_ADD if c["fn"] == "add" else L.EW_MUL, s["A"], s["B"])
        return [C.ptr, C.idx, C.val]
    if op == "ewise_reduce":
        return fg.ewise_reduce(c["dims"], s["A"], B=s["B"])
    if op == "spgemm":
        C = device.spgemm(s["A"], s["B"])
        return [C.ptr, C.idx, C.val]
    if op == "pagerank":
        return examples.pagerank(s["edges"], nsteps=c["steps"]).ddata
    x, _ = cg.cg_solve(s["A"], s["b"], precision=c["precision"], accumulate=c["accumulate"], rtol=c["rtol"],
                       Alow=s["low"])
    return x


# ---------------------------------------------------------------- compulsory work


def work(case):
    c, op = case, case["op"]
    if op == "cg":
        # per iteration: the matrix once, and the vectors' reads and writes of
        # three fused steps; about 3.3 iterations per grid line at 1e-10
        n = c["grid"] ** 2
        it = 3.3 * c["grid"] * (1.0 if c["rtol"] < 1e-9 else 0.8)
        return {"bytes": it * (5 * n * (2 + _size(c["precision"])) + 4 * n + 80 * n), "flops": it * 22 * n}
    if op == "spgemm" and c["grid"]:
        n = c["grid"] ** 2
        return {"bytes": 5 * n * (4 + _size(c["val"])) + 4 * n + 13 * n * (4 + _size(c["val"])) + 4 * n,
                "flops": 2 * 25 * n}
    m = c["m"]
    nnz = m * c["mean"]
    if op == "spgemm":
        prod = m * c["mean"] ** 2
        return {"bytes": 2 * (nnz * (4 + _size(c["val"])) + 4 * m) + prod * (4 + _size(c["val"])) + 4 * m,
                "flops": 2 * prod}
    if op == "pagerank":
        nnz += m
        step = nnz * 12 + 4 * m + 5 * 8 * m
        return {"bytes": 3 * nnz * 12 + c["steps"] * step, "flops": c["steps"] * (2 * nnz + 2 * m)}
    n, v = c["n"], _size(c["val"])
    mat = 4 * (m + 1) + nnz * (4 + v)
    if op == "spmv":
        e = _size(c["vec"])
        return {"bytes": mat + e * n + e * m * (2 if c["accumulate"] else 1), "flops": 2 * nnz}
    if op == "spmm":
        e = _size(c["vec"])
        return {"bytes": mat + e * c["k"] * (m + n), "flops": 2 * nnz * c["k"]}
    if op == "sddmm":
        return {"bytes": mat + v * c["k"] * (m + n) + v * nnz, "flops": 2 * nnz * c["k"]}
    if op == "ewise":
        return {"bytes": 2 * mat + 8 * (m + 1) + (1.5 if c["fn"] == "add" else 0.5) * nnz * (4 + v), "flops": nnz}
    return {"bytes": 2 * mat + v * {0: 1, 1: n, 2: m}[c["dims"]], "flops": 2 * nnz}


# ---------------------------------------------------------------- results in 64 bits


def _triplets(A):
    """Row, column (from 0) and FP64 (or Int64) value of every stored entry."""
    nf = A.ptr.numel() - 1
    fib = torch.repeat_interleave(torch.arange(nf, device="cuda"), (A.ptr[1:] - A.ptr[:-1]).long())
    coord = A.idx.long() - 1
    i, j = (fib, coord) if A.orient == "csr" else (coord, fib)
    return i, j, A.val if not A.val.dtype.is_floating_point else A.val.double()


def _wide(t):
    return t.double() if t.is_floating_point() else t.long()


def _keyed(A):
    nf, ne = (A.nrows, A.ncols) if A.orient == "csr" else (A.ncols, A.nrows)
    fib = torch.repeat_interleave(torch.arange(nf, device="cuda"), (A.ptr[1:] - A.ptr[:-1]).long())
    return fib * ne + A.idx.long() - 1, nf, ne


def _compressed(key, nf, ne, base):
    fib = torch.div(key, ne, rounding_mode="floor")
    ptr = torch.full((nf + 1,), base, dtype=torch.int64, device="cuda")
    ptr[1:] += torch.cumsum(torch.bincount(fib, minlength=nf), 0)
    return ptr, (key - fib * ne + base).to(torch.int32)


def exact(case, seed):
    c, op = case, case["op"]
    s = prepare({**c, "route": "call"} if op == "spmm" else c, seed)
    if op == "spmv":
        i, j, a = _triplets(s["A"])
        x = _wide(s["x"])
        if c["semiring"] == "plus_times":
            y = _wide(s["y0"]) if c["accumulate"] else torch.zeros(c["m"], dtype=x.dtype, device="cuda")
            return y.index_add_(0, i, _wide(a) * x[j])
        low = c["semiring"] == "min_plus"
        if x.is_floating_point():
            ident = math.inf if low else -math.inf
        else:
            info = torch.iinfo(s["x"].dtype)
            ident = info.max if low else info.min
        y = _wide(s["y0"]) if c["accumulate"] else torch.full((c["m"],), ident, dtype=x.dtype, device="cuda")
        return y.scatter_reduce_(0, i, _wide(a) + x[j], "amin" if low else "amax")
    if op == "spmm":
        i, j, a = _triplets(s["A"])
        out = torch.zeros((c["m"], c["k"]), dtype=torch.float64, device="cuda")
        for k in range(0, c["k"], 16):
            out[:, k:k + 16] = torch.zeros((c["m"], min(16, c["k"] - k)), dtype=torch.float64, device="cuda").index_add_(
                0, i, s["B"][:, k:k + 16].double()[j] * a[:, None])
        return out
    if op == "sddmm":
        i, j, a = _triplets(s["A"])
        step = 1 << 20
        return torch.cat([a[e:e + step] * (s["X"][i[e:e + step]].double() * s["Y"][j[e:e + step]].double()).sum(1)
                          for e in range(0, max(1, a.numel()), step)])
    if op == "ewise":
        (ka, nf, ne), (kb, _, _) = _keyed(s["A"]), _keyed(s["B"])
        va, vb = _wide(s["A"].val), _wide(s["B"].val)
        if c["fn"] == "add":
            key, at = torch.unique(torch.cat([ka, kb]), return_inverse=True)
            val = torch.zeros(key.numel(), dtype=va.dtype, device="cuda").index_add_(0, at, torch.cat([va, vb]))
        else:
            pos = torch.searchsorted(kb, ka).clamp_(max=max(0, kb.numel() - 1))
            hit = kb[pos] == ka
            key, val = ka[hit], va[hit] * vb[pos[hit]]
        return [*_compressed(key, nf, ne, 0), val]
    if op == "ewise_reduce":
        (ka, nf, ne), (kb, _, _) = _keyed(s["A"]), _keyed(s["B"])
        pos = torch.searchsorted(kb, ka).clamp_(max=max(0, kb.numel() - 1))
        hit = kb[pos] == ka
        prod = s["A"].val.double()[hit] * s["B"].val.double()[pos[hit]]
        i, j, _ = _triplets(s["A"])
        if c["dims"] == 0:
            return prod.sum().reshape(1)
        at = (i if c["dims"] == 2 else j)[hit]
        return torch.zeros(c["m"] if c["dims"] == 2 else c["n"], dtype=torch.float64, device="cuda").index_add_(0, at, prod)
    if op == "spgemm":
        i, k, a = _triplets(s["A"])
        B = s["B"]
        deg = (B.ptr[1:] - B.ptr[:-1]).long()[k]
        e = torch.repeat_interleave(torch.arange(k.numel(), device="cuda"), deg)
        first = torch.cumsum(deg, 0) - deg
        p = (B.ptr.long() - 1)[k][e] + torch.arange(e.numel(), device="cuda") - first[e]
        key, at = torch.unique(i[e] * B.ncols + B.idx.long()[p] - 1, return_inverse=True)
        val = torch.zeros(key.numel(), dtype=torch.float64, device="cuda").index_add_(0, at, a[e] * B.val.double()[p])
        ptr, idx = _compressed(key, s["A"].nrows, B.ncols, 1)
        return [ptr.to(torch.int32), idx, val]
    if op == "pagerank":
        n, damp = c["m"], 0.85
        E = s["E"]
        deg = (E.ptr[1:] - E.ptr[:-1]).double()
        j = torch.repeat_interleave(torch.arange(n, device="cuda"), deg.long())
        i, w = E.idx.long() - 1, 1.0 / deg[j]
        r = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
        for _ in range(c["steps"]):
            r = (1 - damp) / n + damp * torch.zeros_like(r).index_add_(0, i, w * r[j])
        return r
    # the 5-point matrix in the sine basis: eigenvalues 4 - 2 cos - 2 cos
    N = c["grid"]
    t = torch.arange(1, N + 1, dtype=torch.float64, device="cuda") * (math.pi / (N + 1))
    S = torch.sin(t[:, None] * torch.arange(1, N + 1, dtype=torch.float64, device="cuda")) * math.sqrt(2 / (N + 1))
    lam = 2 - 2 * torch.cos(t)
    X = S @ s["b"].reshape(N, N) @ S / (lam[:, None] + lam[None, :])
    return (S @ X @ S).reshape(-1)
