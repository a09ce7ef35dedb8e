"""Performance cases: the work a program gives this library, through its public entry points.

`listed()` names twelve calls that stand for the whole range: the smallest products, where the call itself is the
cost, ordinary and ragged ones, and the largest; every semiring and element type of the benchmark configurations
(cuasr_b200/workloads.py); products with and without the optional workspace; the split-K, path-tracking, shortest-path
and host-buffer entry points.  `draw(rng)` makes further calls of the same ranges.
"""
from __future__ import annotations

import math

import torch

from cuasr_b200 import (Arguments, DType, HostSrgemm, Layout, RINGS, Srgemm, SrgemmSplitKParallel, Status, identity,
                        srgemm_path)
from cuasr_b200 import apsp

TORCH_DTYPE = {"f32": torch.float32, "f64": torch.float64, "s32": torch.int32, "u32": torch.int32}
DTYPE = {"f32": DType.F32, "f64": DType.F64, "s32": DType.S32, "u32": DType.U32}
LAYOUT = {"c": Layout.COLUMN_MAJOR, "r": Layout.ROW_MAJOR}

# (ring, element type) pairs of the benchmark configurations
PAIRS = [("minimum_plus", "f32"), ("maximum_plus", "f32"), ("minimum_plus", "f64"), ("maximum_plus", "f64"),
         ("maximum_minimum", "f32"), ("plus_multiplies", "f64"), ("minimum_plus", "s32"), ("bit_xor_bit_and", "u32")]


def product(name, ring, dtype, m, n, k, layouts="ccc", pad=0, workspace=False):
    """One call of Srgemm.  layouts: of A, B and C/D (c = column-major, r = row-major).  pad: elements added to the
    leading dimensions of A and B.  workspace: hand over the optional workspace."""
    case = {"kind": "product", "ring": ring, "dtype": dtype, "m": m, "n": n, "k": k, "layouts": layouts, "pad": pad,
            "workspace": workspace}
    return dict(case, name=name) if name else case


def listed():
    return [
        # The smallest call: a product of a few microseconds inside a loop of a host program, or one block of a
        # blocked algorithm.  What counts is the call.
        product("minplus_f32_64", "minimum_plus", "f32", 64, 64, 64),
        # The reference's own CPU-runnable configuration, with the workspace the library asks for.
        product("minplus_f32_512", "minimum_plus", "f32", 512, 512, 512, workspace=True),
        # An ordinary product as a graph program has it: odd sizes, so that no storage line is 16-byte aligned, and
        # no workspace.
        product("minplus_f32_ragged", "minimum_plus", "f32", 1021, 765, 1533),
        # The headline benchmark.
        product("minplus_f32_8192", "minimum_plus", "f32", 8192, 8192, 8192, workspace=True),
        # Double-precision distances over weighted adjacency matrices (10 % of the edges present, +inf elsewhere).
        product("minplus_f64_4096", "minimum_plus", "f64", 4096, 4096, 4096, workspace=True),
        # Bottleneck paths.
        product("maxmin_f32_4096", "maximum_minimum", "f32", 4096, 4096, 4096, workspace=True),
        # The ordinary product in double precision, row-major, at a size that is no multiple of any tile.
        product("plustimes_f64_1500", "plus_multiplies", "f64", 1500, 1500, 1500, layouts="rrr"),
        # GF(2) words, a middle size.
        product("xorand_u32_1024", "bit_xor_bit_and", "u32", 1024, 1024, 1024),
        # A long contraction with a small output, cut along K.
        {"name": "splitk_minplus_f32", "kind": "splitk", "m": 256, "n": 256, "k": 262144, "slices": 32},
        # Distances together with the vertex each of them goes through.
        {"name": "path_minplus_f32_2048", "kind": "path", "m": 2048, "n": 2048, "k": 2048},
        # All-pairs shortest paths of a sparse graph with the blocked Floyd-Warshall solve.
        {"name": "apsp_fw_2000", "kind": "apsp", "n": 2000, "algorithm": apsp.BLOCKED_FLOYD_WARSHALL},
        # Matrices that live in host memory: copies in, product, copy out.
        {"name": "host_minplus_f32_4096", "kind": "host", "m": 4096, "n": 4096, "k": 4096},
    ]


def _log(rng, lo, hi):
    """A whole number from [lo, hi], spread evenly over its logarithm; odd ones as likely as even ones."""
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["product"] * 8 + ["splitk", "path", "apsp", "host"])
    if kind == "product":
        ring, dtype = rng.choice(PAIRS)
        m, n, k = (_log(rng, 32, 4096) for _ in range(3))
        if rng.random() < 0.4:       # sizes whose storage lines are 16-byte aligned
            m, n, k = (min(4096, (v + 3) // 4 * 4) for v in (m, n, k))
        return product(None, ring, dtype, m, n, k, "".join(rng.choice("cr") for _ in range(3)),
                       rng.choice((0, 0, 0, 1, 4)), rng.random() < 0.5)
    if kind == "splitk":
        m, n = (_log(rng, 32, 512) for _ in range(2))
        return {"kind": kind, "m": m, "n": n, "k": _log(rng, 8192, 524288), "slices": rng.choice((8, 16, 32, 64))}
    if kind == "path":
        return {"kind": kind, "m": _log(rng, 128, 3072), "n": _log(rng, 128, 3072), "k": _log(rng, 128, 3072)}
    if kind == "apsp":
        return {"kind": kind, "n": _log(rng, 200, 3000),
                "algorithm": rng.choice((apsp.REPEATED_SQUARING, apsp.BLOCKED_FLOYD_WARSHALL))}
    return {"kind": kind, "m": 128 * _log(rng, 4, 32), "n": 128 * _log(rng, 4, 32), "k": 128 * _log(rng, 4, 32)}


# ---- inputs ---------------------------------------------------------------------------------------------------
def _values(g, count, ring, dtype):
    """Operands as the benchmark configurations fill them: uniform weights for float min-plus and max-plus (sparse
    weighted adjacency for double precision), [0, 1) for max-min, [-1, 1) for plus-times, whole numbers below 1000,
    random words."""
    dev = torch.device("cuda")
    if dtype == "u32":
        return torch.randint(-2 ** 31, 2 ** 31, (count,), generator=g, device=dev, dtype=torch.int64).to(torch.int32)
    if dtype == "s32":
        return torch.randint(0, 1000, (count,), generator=g, device=dev, dtype=torch.int32)
    x = torch.rand(count, generator=g, device=dev, dtype=TORCH_DTYPE[dtype])
    if ring == "plus_multiplies":
        return x.mul_(2).sub_(1)
    if ring == "maximum_minimum":
        return x
    if dtype == "f64":
        absent = math.inf if ring == "minimum_plus" else -math.inf
        x.mul_(999).add_(1)
        present = torch.rand(count, generator=g, device=dev) < 0.1
        return torch.where(present, x, absent)
    return x.mul_(100)


def _lead(layout, rows, cols):
    """(contiguous extent, number of storage lines) of a rows x cols matrix."""
    return (rows, cols) if layout == "c" else (cols, rows)


def _scalars(ring, dtype):
    """Additive identity, alpha and beta of D = (alpha (x) A B) (+) (beta (x) C): infinities where the type has them."""
    add, mul = RINGS[ring]
    true_inf = dtype in ("f32", "f64")
    one = identity(mul, DTYPE[dtype], true_infinity=true_inf)
    return identity(add, DTYPE[dtype], true_infinity=true_inf), one, one


def _operator(cls, case, ring, dtype, layouts):
    add, mul = RINGS[ring]
    zero, _, _ = _scalars(ring, dtype)
    return cls(add, mul, DTYPE[dtype], *[LAYOUT[c] for c in layouts], add_identity=zero)


def _checked(status):
    if status != Status.kSuccess:
        raise RuntimeError(f"the library refused the call: {status!r}")


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    dev = torch.device("cuda")
    s = {"case": case}
    kind = case["kind"]
    if kind in ("product", "splitk"):
        splitk = kind == "splitk"
        ring, dtype, layouts, pad = (("minimum_plus", "f32", "rcr", 0) if splitk else
                                     (case["ring"], case["dtype"], case["layouts"], case["pad"]))
        m, n, k = case["m"], case["n"], case["k"]
        s["op"] = op = _operator(SrgemmSplitKParallel if splitk else Srgemm, case, ring, dtype, layouts)
        zero, s["alpha"], s["beta"] = _scalars(ring, dtype)
        for key, layout, rows, cols in (("A", layouts[0], m, k), ("B", layouts[1], k, n)):
            extent, lines = _lead(layout, rows, cols)
            s[key], s["ld" + key] = _values(g, (extent + pad) * lines, ring, dtype), extent + pad
        s["ldC"] = _lead(layouts[2], m, n)[0]
        s["C"] = torch.full((m * n,), zero.item(), dtype=TORCH_DTYPE[dtype], device=dev)
        s["D"] = torch.empty_like(s["C"])
        args = _arguments(s)
        need = op.get_workspace_size(args)
        if not splitk and case["workspace"]:
            need = op.get_optional_workspace_size(args)
        s["workspace"] = torch.empty(need, dtype=torch.uint8, device=dev) if need else None
    elif kind == "path":
        m, n, k = case["m"], case["n"], case["k"]
        s["op"] = _operator(Srgemm, case, "minimum_plus", "f32", "ccc")
        s["A"], s["B"] = _values(g, m * k, "minimum_plus", "f32"), _values(g, k * n, "minimum_plus", "f32")
        s["dist"] = torch.empty(m * n, dtype=torch.float32, device=dev)
        s["parent"] = torch.empty(m * n, dtype=torch.int32, device=dev)
    elif kind == "apsp":
        # a random directed graph: on average ten edges leave a vertex, whole weights from 1 to 100
        n = case["n"]
        w = torch.randint(1, 101, (n, n), generator=g, device=dev).float()
        absent = torch.rand(n, n, generator=g, device=dev) >= 10.0 / n
        w[absent] = math.inf
        w.fill_diagonal_(0)
        s["graph"], s["D"] = w.reshape(-1), torch.empty(n * n, dtype=torch.float32, device=dev)
        need = apsp.device_solve_workspace_size(DType.F32, case["algorithm"], n)
        s["workspace"] = torch.empty(need, dtype=torch.uint8, device=dev)
    else:
        m, n, k = case["m"], case["n"], case["k"]
        op = _operator(Srgemm, case, "minimum_plus", "f32", "ccc")
        for key, count in (("A", m * k), ("B", k * n), ("C", m * n)):
            s[key] = torch.empty(count, dtype=torch.float32, pin_memory=True)
            s[key].copy_(_values(g, count, "minimum_plus", "f32") * (2 if key == "C" else 1))
        s["D"] = torch.empty(m * n, dtype=torch.float32, pin_memory=True)
        s["pipeline"] = HostSrgemm(op, m, n, k, 0.0, 0.0, dev)
    return s


def _arguments(s):
    c = s["case"]
    return Arguments((c["m"], c["n"], c["k"]), (s["A"], s["ldA"]), (s["B"], s["ldB"]), (s["C"], s["ldC"]),
                     (s["D"], s["ldC"]), (s["alpha"], s["beta"]), c.get("slices", 1))


# ---- one pass -------------------------------------------------------------------------------------------------
def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind in ("product", "splitk"):
        _checked(s["op"](_arguments(s), s["workspace"]))
        return s["D"]
    if kind == "path":
        m, n, k = c["m"], c["n"], c["k"]
        s["dist"].fill_(math.inf)
        s["parent"].fill_(-1)
        _checked(srgemm_path(s["op"], (m, n, k), (s["A"], m), (s["B"], k), (s["dist"], m), (s["parent"], m)))
        return s["dist"], s["parent"]
    if kind == "apsp":
        s["D"].copy_(s["graph"])
        _checked(apsp.device_solve(s["D"], c["n"], DType.F32, c["algorithm"], workspace=s["workspace"]))
        return s["D"]
    s["pipeline"](s["A"], s["B"], s["C"], s["D"])
    return s["D"]


def work(case):
    """Each operand read once, each result written once; two semiring operations per product."""
    if case["kind"] == "apsp":
        n = case["n"]
        return {"bytes": 2 * 4 * n * n, "flops": 2.0 * n ** 3}
    m, n, k = case["m"], case["n"], case["k"]
    es = 8 if case.get("dtype") == "f64" else 4
    # a path product has no input but the operands and writes distances and vertices; the others read C
    return {"bytes": es * (m * k + k * n + 2 * m * n), "flops": 2.0 * m * n * k}


def tolerance(case):
    """Sums of two values rounded once, minima, maxima, words, whole numbers: nothing depends on an order.  The double
    precision sums of plus-times do."""
    return {"rel": 1e-13} if case.get("ring") == "plus_multiplies" else "exact"
