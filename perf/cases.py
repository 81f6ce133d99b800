"""Performance cases of the framework's public entry points.

Every case is one call (or the few calls of one step) that a program makes
through ``alp_b200.device`` / ``alp_b200._abi``, on the kinds of matrices that
the benchmark and the tests use: R-MAT graphs, 27-point and 5-point stencils.
Inputs are made on the GPU from the seed with plain torch; ``exact`` gives the
same results from plain torch in 64 bits.

Kinds
  mxv           one matrix-vector product over a semiring, dense or with sparse
                vectors and masks (a graph traversal step)
  cg            one conjugate-gradient solve of a 27-point system
  cg_grad       a differentiated solve: forward, adjoint and dL/dA
  batched_cg    many 5-point Poisson systems of uneven size, one launch
  pagerank      one PageRank solve on a graph whose plan and scratch are kept
  hpcg          a fixed number of HPCG iterations (multigrid-preconditioned CG)
  ppr           personalised PageRank: forward, adjoint, edge-weight gradient
  level1        the vector steps of one CG iteration, composed by the caller
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from alp_b200 import _abi as abi
from alp_b200 import device as dev

F64 = torch.float64


# ------------------------------------------------------------------ cases --
def listed() -> list[dict]:
    return [
        # the benchmark's headline: a dense product on the scale-22 graph, its
        # plan tuned once and kept
        {"name": "mxv_f64_rmat22", "kind": "mxv", "ring": "plus_times_f64", "graph": "rmat",
         "m": 1 << 22, "n": 1 << 22, "edge_factor": 16, "tuned": True, "frontier": 0.0,
         "visited": 0.0},
        # a small graph, as the smoke program's: the cost of a call
        {"name": "mxv_f64_rmat12", "kind": "mxv", "ring": "plus_times_f64", "graph": "rmat",
         "m": 1 << 12, "n": 1 << 12, "edge_factor": 16, "tuned": False, "frontier": 0.0,
         "visited": 0.0},
        # the product inside a hand-written stencil solver, ragged grid
        {"name": "mxv_f64_27pt_ragged", "kind": "mxv", "ring": "plus_times_f64",
         "graph": "27pt", "m": 129 * 127 * 131, "n": 129 * 127 * 131, "side": 129,
         "tuned": False, "frontier": 0.0, "visited": 0.0},
        # one breadth-first step: sparse frontier in, sparse output, visited
        # vertices masked out (structural, inverted)
        {"name": "mxv_bool_bfs", "kind": "mxv", "ring": "lor_land_bool", "graph": "rmat",
         "m": 1000003, "n": 1000003, "edge_factor": 16, "tuned": False, "frontier": 0.05,
         "visited": 0.3},
        # one relaxation step of shortest paths: distances dense, the vertices
        # that changed last round sparse
        {"name": "mxv_i32_sssp", "kind": "mxv", "ring": "min_plus_i32", "graph": "rmat",
         "m": 500009, "n": 500009, "edge_factor": 16, "tuned": False, "frontier": 0.2,
         "visited": 0.0},
        # the reference's own CG configuration
        {"name": "cg_27pt_32", "kind": "cg", "nx": 32, "ny": 32, "nz": 32},
        # the benchmark's differentiated CG
        {"name": "cg_grad_27pt_64", "kind": "cg_grad", "nx": 64, "ny": 64, "nz": 64},
        # the benchmark's batch: 256 systems, sides log-uniform in [32, 512]
        {"name": "batched_cg_256", "kind": "batched_cg", "systems": 256, "lo": 32, "hi": 512},
        # PageRank on a graph of a million pages
        {"name": "pagerank_1m", "kind": "pagerank", "n": 1000003, "edge_factor": 16},
        # HPCG on 64^3 with three coarser levels, eight right-hand sides
        {"name": "hpcg_64_8rhs", "kind": "hpcg", "nx": 64, "ny": 64, "nz": 64, "levels": 3,
         "nrhs": 8, "iterations": 10},
        # 32 seeds on a graph of 131,072 vertices, forward and backward
        {"name": "ppr_rmat17_32", "kind": "ppr", "n": 1 << 17, "edge_factor": 16, "seeds": 32},
        # level-1 steps on a vector of about the HPCG 100^3 size
        {"name": "level1_1m", "kind": "level1", "n": 1000003},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["mxv", "mxv", "mxv", "mxv", "cg", "cg_grad", "batched_cg", "pagerank",
                       "hpcg", "ppr", "level1"])
    if kind == "mxv":
        graph = rng.choice(["rmat", "rmat", "27pt", "5pt"])
        if graph == "27pt":
            nx, ny, nz = (_log_int(rng, 12, 140) for _ in range(3))
            return {"kind": kind, "ring": "plus_times_f64", "graph": graph, "m": nx * ny * nz,
                    "n": nx * ny * nz, "side": nx, "ny": ny, "tuned": rng.random() < 0.5,
                    "frontier": 0.0, "visited": 0.0}
        if graph == "5pt":
            side = _log_int(rng, 32, 2000)
            return {"kind": kind, "ring": "plus_times_f64", "graph": graph, "m": side * side,
                    "n": side * side, "side": side, "tuned": rng.random() < 0.5,
                    "frontier": 0.0, "visited": 0.0}
        ring = rng.choice(["plus_times_f64", "min_plus_i32", "lor_land_bool"])
        m = _log_int(rng, 1000, 1 << 21)
        n = m if rng.random() < 0.7 else _log_int(rng, max(1000, m // 4), min(1 << 21, 4 * m))
        sparse = ring != "plus_times_f64" and rng.random() < 0.6
        return {"kind": kind, "ring": ring, "graph": graph, "m": m, "n": n,
                "edge_factor": rng.choice([8, 16]), "tuned": not sparse and rng.random() < 0.3,
                "frontier": rng.choice([0.01, 0.05, 0.2]) if sparse else 0.0,
                "visited": rng.choice([0.1, 0.3, 0.6])
                if sparse and ring == "lor_land_bool" else 0.0}
    if kind == "cg":
        return {"kind": kind, "nx": _log_int(rng, 10, 80), "ny": _log_int(rng, 10, 80),
                "nz": _log_int(rng, 10, 80)}
    if kind == "cg_grad":
        return {"kind": kind, "nx": _log_int(rng, 10, 64), "ny": _log_int(rng, 10, 64),
                "nz": _log_int(rng, 10, 64)}
    if kind == "batched_cg":
        lo = _log_int(rng, 8, 64)
        return {"kind": kind, "systems": _log_int(rng, 4, 256), "lo": lo,
                "hi": _log_int(rng, 2 * lo, 512)}
    if kind == "pagerank":
        return {"kind": kind, "n": _log_int(rng, 4000, 1000000), "edge_factor": rng.choice([8, 16])}
    if kind == "hpcg":
        levels = rng.choice([1, 2, 3])
        unit = 4 << (levels - 1)
        side = [2 * unit * rng.randint(1, 32 // unit) for _ in range(3)]
        return {"kind": kind, "nx": side[0], "ny": side[1], "nz": side[2], "levels": levels,
                "nrhs": rng.choice([1, 2, 4, 8]), "iterations": 10}
    if kind == "ppr":
        return {"kind": kind, "n": _log_int(rng, 2000, 120000), "edge_factor": rng.choice([8, 16]),
                "seeds": rng.choice([1, 5, 16, 32])}
    return {"kind": kind, "n": _log_int(rng, 1000, 16000000)}


# ----------------------------------------------------------------- inputs --
def _gen(seed: int) -> torch.Generator:
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _crs_from_keys(key, m):
    """offsets and column indices from sorted unique (row << 32 | col) keys"""
    rows = key >> 32
    offsets = torch.zeros(m + 1, dtype=torch.int64, device="cuda")
    offsets[1:] = torch.bincount(rows, minlength=m)
    torch.cumsum(offsets, 0, out=offsets)
    return offsets, (key & 0xFFFFFFFF).to(torch.int32)


def _rmat(m: int, n: int, edge_factor: int, g):
    """R-MAT a/b/c/d = .57/.19/.19/.05, cut to m x n, duplicates merged"""
    scale = max(1, (max(m, n) - 1).bit_length())
    count = edge_factor * max(m, n)
    row = torch.zeros(count, dtype=torch.int64, device="cuda")
    col = torch.zeros_like(row)
    for _ in range(scale):
        h = torch.rand(count, generator=g, device="cuda")
        row = 2 * row + (h >= 0.76)
        col = 2 * col + (((h >= 0.57) & (h < 0.76)) | (h >= 0.95))
    key = (row << 32) | col
    key = key[(row < m) & (col < n)]
    del row, col, h
    return _crs_from_keys(torch.unique(key), m)


def _stencil(sizes):
    """Box stencil of halo 1 on the grid `sizes` (dimension 0 fastest), columns
    decreasing in each row (the order the framework's builder stores)"""
    nx, ny, nz = sizes
    m = nx * ny * nz
    i = torch.arange(m, device="cuda")
    x, y, z = i % nx, (i // nx) % ny, i // (nx * ny)
    cols, ok = [], []
    for dz in (1, 0, -1):
        for dy in (1, 0, -1):
            for dx in (1, 0, -1):
                ok.append((x + dx >= 0) & (x + dx < nx) & (y + dy >= 0) & (y + dy < ny) &
                          (z + dz >= 0) & (z + dz < nz))
                cols.append(i + dx + nx * (dy + ny * dz))
    return _pack(m, cols, ok)


def _poisson(sides):
    """5-point stencils on L x L grids, one block per side, columns increasing"""
    L = torch.tensor(sides, device="cuda")
    rows = L * L
    start = torch.cumsum(rows, 0) - rows
    s = torch.repeat_interleave(torch.arange(len(sides), device="cuda"), rows)
    i = torch.arange(int(rows.sum()), device="cuda")
    Li, r = L[s], i - start[s]
    x, y = r % Li, r // Li
    cols = [i - Li, i - 1, i, i + 1, i + Li]
    ok = [y > 0, x > 0, torch.ones_like(x, dtype=torch.bool), x < Li - 1, y < Li - 1]
    offsets, indices = _pack(len(i), cols, ok)
    return offsets, indices, s


def _pack(m, cols, ok):
    mask = torch.stack(ok, 1)
    offsets = torch.zeros(m + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(mask.sum(1), 0, out=offsets[1:])
    return offsets, torch.stack(cols, 1)[mask].to(torch.int32)


def _row_index(offsets):
    m = len(offsets) - 1
    return torch.repeat_interleave(torch.arange(m, device="cuda"), offsets[1:] - offsets[:-1])


def _transpose(offsets, indices, values, n):
    rows = _row_index(offsets)
    order = torch.sort(indices, stable=True).indices
    t = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    t[1:] = torch.cumsum(torch.bincount(indices, minlength=n), 0)
    return t, rows[order].to(torch.int32), values[order]


def _sym_dd(offsets, indices, g):
    """symmetric off-diagonals -U(0.5, 1.5), diagonal 1.05 times the row sum"""
    rows, cols = _row_index(offsets), indices.to(torch.int64)
    m = len(offsets) - 1
    w = torch.rand(m, generator=g, device="cuda", dtype=F64)
    v = -(0.5 + torch.frac(w[torch.minimum(rows, cols)] + 1.7 * w[torch.maximum(rows, cols)]))
    diag = rows == cols
    v[diag] = 0.0
    total = torch.zeros(m, dtype=F64, device="cuda").index_add_(0, rows, -v)
    v[diag] = 1.05 * total[rows[diag]]
    return v


RINGS = {"plus_times_f64": (abi.RING_PLUS_TIMES_F64, abi.FP64, F64),
         "min_plus_i32": (abi.RING_MIN_PLUS_I32, abi.INT32, torch.int32),
         "lor_land_bool": (abi.RING_LOR_LAND_BOOL, abi.BOOL, torch.uint8)}
INF = 2 ** 31 - 1


def _mxv_inputs(case, seed):
    g = _gen(seed)
    m, n = case["m"], case["n"]
    if case["graph"] == "rmat":
        offsets, indices = _rmat(m, n, case["edge_factor"], g)
    elif case["graph"] == "27pt":
        nx = case["side"]
        ny = case.get("ny", 127)
        offsets, indices = _stencil((nx, ny, m // (nx * ny)))
    else:
        offsets, indices, _ = _poisson([case["side"]])
    nnz = len(indices)
    if case["ring"] == "plus_times_f64":
        values = torch.rand(nnz, generator=g, device="cuda", dtype=F64)
        v = torch.rand(n, generator=g, device="cuda", dtype=F64)
        u = torch.rand(m, generator=g, device="cuda", dtype=F64)
    elif case["ring"] == "min_plus_i32":
        values = torch.randint(1, 101, (nnz,), generator=g, device="cuda", dtype=torch.int32)
        v = torch.randint(0, 1001, (n,), generator=g, device="cuda", dtype=torch.int32)
        u = torch.randint(0, 1001, (m,), generator=g, device="cuda", dtype=torch.int32)
        u[torch.rand(m, generator=g, device="cuda") < 0.3] = INF
    else:
        values = None
        v = torch.ones(n, dtype=torch.uint8, device="cuda") if case["frontier"] else \
            (torch.rand(n, generator=g, device="cuda") < 0.5).to(torch.uint8)
        u = torch.zeros(m, dtype=torch.uint8, device="cuda")
    d = {"offsets": offsets, "indices": indices, "values": values, "u": u, "v": v}
    if case["frontier"]:
        d["v_assigned"] = (torch.rand(n, generator=g, device="cuda") <
                           case["frontier"]).to(torch.uint8)
    if case["visited"]:
        d["mask_assigned"] = (torch.rand(m, generator=g, device="cuda") <
                              case["visited"]).to(torch.uint8)
        d["mask"] = torch.ones(m, dtype=torch.uint8, device="cuda")
    return d


def _cg_inputs(case, seed):
    """diagonal 26, off-diagonals -1; b = A x for a random x"""
    offsets, indices = _stencil((case["nx"], case["ny"], case["nz"]))
    n = len(offsets) - 1
    values = torch.where(_row_index(offsets) == indices, 26.0, -1.0).to(F64)
    x = torch.randn(n, generator=_gen(seed), device="cuda", dtype=F64)
    return offsets, indices, values, _spmv(offsets, indices, values, x), x


def _cg_grad_inputs(case, seed):
    g = _gen(seed)
    offsets, indices = _stencil((case["nx"], case["ny"], case["nz"]))
    values = _sym_dd(offsets, indices, g)
    n = len(offsets) - 1
    b = torch.randn(n, generator=g, device="cuda", dtype=F64)
    target = torch.randn(n, generator=g, device="cuda", dtype=F64)
    return offsets, indices, values, b, target


def _batch_inputs(case, seed):
    k = case["systems"]
    sides = np.exp(np.random.default_rng(2024).uniform(math.log(case["lo"]), math.log(case["hi"]), k))
    sides = np.round(sides).astype(int)     # the batch's sizes are the case's own
    shifts = np.random.default_rng(seed).uniform(0.01, 1.0, k)
    offsets, indices, seg = _poisson(sides.tolist())
    rows = _row_index(offsets)
    shift = torch.from_numpy(shifts).cuda()
    values = torch.where(rows == indices, 4.0 + shift[seg[rows]], -1.0)
    b = torch.randn(len(seg), generator=_gen(seed), device="cuda", dtype=F64)
    return sides, shifts, offsets, indices, values, b


def _ppr_inputs(case, seed):
    g = _gen(seed)
    n, S = case["n"], case["seeds"]
    offsets, indices = _rmat(n, n, case["edge_factor"], _gen(42))   # edges as the case's own
    weights = torch.rand(len(indices), generator=g, device="cuda", dtype=F64)
    seeds = np.random.default_rng(seed).integers(0, n, S)
    dl_dx = torch.randn(n * S, generator=g, device="cuda", dtype=F64)
    return offsets, indices, weights, seeds, dl_dx


# ---------------------------------------------------------------- prepare --
class _Handle:
    """a solver handle and the tensors it holds by reference"""

    def __init__(self, create, destroy, *args, keep=()):
        self.h = C.c_void_p()
        self.destroy = destroy
        self.keep = keep
        abi.call(create, C.byref(self.h), *args)

    def __del__(self):
        getattr(abi.lib(), self.destroy)(self.h)


def prepare(case: dict, seed: int) -> dict:
    abi.call("alpb_init", torch.cuda.current_device())
    return {"kind": case["kind"], **globals()["_prepare_" + case["kind"]](case, seed)}


def _prepare_mxv(case, seed):
    d = _mxv_inputs(case, seed)
    ring, vtype, dtype = RINGS[case["ring"]]
    A = dev.CRS(case["m"], case["n"], len(d["indices"]), d["offsets"], d["indices"], d["values"],
                abi.VOID if d["values"] is None else vtype)
    plan = dev.Plan(A)
    if case["tuned"]:
        plan.autotune(ring, d["v"], torch.zeros(A.m, dtype=dtype, device="cuda"))
    st = {"ring": ring, "A": A, "u": d["u"], "v": d["v"], "plan": plan}
    if case["frontier"]:
        st["v_assigned"] = d["v_assigned"]
        st["v_count"] = int(d["v_assigned"].sum())
    if case["visited"]:
        st["mask"], st["mask_assigned"] = d["mask"], d["mask_assigned"]
        st["mask_count"] = int(d["mask_assigned"].sum())
        st["u_assigned"] = torch.zeros(A.m, dtype=torch.uint8, device="cuda")
        st["u_nnz"] = torch.zeros(1, dtype=torch.int64, device="cuda")
    return st


def _prepare_cg(case, seed):
    offsets, indices, values, b, x = _cg_inputs(case, seed)
    A = dev.CRS(len(b), len(b), len(indices), offsets, indices, values, abi.FP64)
    return {"A": A, "plan": dev.Plan(A, sched=abi.SCHED_MERGE_PATH), "b": b,
            "x": torch.zeros_like(b), "work": torch.empty(4 * len(b), dtype=F64, device="cuda"),
            "iterations": C.c_int64(), "residual": C.c_double()}


def _prepare_cg_grad(case, seed):
    offsets, indices, values, b, target = _cg_grad_inputs(case, seed)
    n = len(b)
    A = dev.CRS(n, n, len(indices), offsets, indices, values, abi.FP64)
    At = dev.CRS(n, n, A.nnz, *_transpose(offsets, indices, values, n), abi.FP64)
    new = lambda k: torch.zeros(k, dtype=F64, device="cuda")  # noqa: E731
    return {"A": A, "At": At, "plan": dev.Plan(A, sched=abi.SCHED_MERGE_PATH),
            "plan_t": dev.Plan(At, sched=abi.SCHED_MERGE_PATH), "b": b, "target": target,
            "x": new(n), "lam": new(n), "grad": new(A.nnz), "work": new(n + 1),
            "loss": C.c_double(), "it": (C.c_int64(), C.c_int64())}


def _prepare_batched_cg(case, seed):
    sides, _, offsets, indices, values, b = _batch_inputs(case, seed)
    seg = torch.from_numpy(np.concatenate([[0], np.cumsum(sides * sides)])).cuda()
    n = len(b)
    h = _Handle("alpb_batched_cg_create", "alpb_batched_cg_destroy", n, len(indices),
                dev.ptr(offsets), dev.ptr(indices), dev.ptr(values), len(sides), dev.ptr(seg),
                dev.stream_ptr(), keep=(offsets, indices, values, seg))
    k = len(sides)
    return {"h": h, "b": b, "x": torch.zeros_like(b), "it": np.zeros(k, np.int64),
            "rr": np.zeros(k), "conv": np.zeros(k, np.int32)}


def _prepare_pagerank(case, seed):
    n = case["n"]
    offsets, indices = _rmat(n, n, case["edge_factor"], _gen(seed))
    ones = torch.ones(len(indices), dtype=F64, device="cuda")
    L = dev.CRS(n, n, len(indices), offsets, indices, ones, abi.FP64)
    LT = dev.CRS(n, n, len(indices), *_transpose(offsets, indices, ones, n), abi.FP64)
    return {"L": L, "LT": LT, "plan": dev.Plan(LT, sched=abi.SCHED_MERGE_PATH),
            "pr": torch.zeros(n, dtype=F64, device="cuda"),
            "work": torch.empty(3 * n, dtype=F64, device="cuda"), "it": C.c_int64(),
            "res": C.c_double()}


def _prepare_hpcg(case, seed):
    h = _Handle("alpb_hpcg_create", "alpb_hpcg_destroy", case["nx"], case["ny"], case["nz"], 26.0,
                -1.0, 27, 4, case["levels"], case["nrhs"], dev.stream_ptr())
    k = case["nx"] * case["ny"] * case["nz"] * case["nrhs"]
    b = torch.randn(k, generator=_gen(seed), device="cuda", dtype=F64)
    return {"h": h, "b": b, "x": torch.zeros_like(b), "max": case["iterations"],
            "it": (C.c_int64 * case["nrhs"])(), "res": (C.c_double * case["nrhs"])()}


def _prepare_ppr(case, seed):
    n, S = case["n"], case["seeds"]
    offsets, indices, weights, seeds, dl_dx = _ppr_inputs(case, seed)
    h = _Handle("alpb_ppr_create", "alpb_ppr_destroy", n, len(indices), dev.ptr(offsets),
                dev.ptr(indices), dev.ptr(weights), S, dev.stream_ptr(),
                keep=(offsets, indices, weights))
    return {"h": h, "seeds": np.ascontiguousarray(seeds, np.int64), "dl_dx": dl_dx,
            "x": torch.zeros(n * S, dtype=F64, device="cuda"), "lam": torch.zeros_like(dl_dx),
            "grad": torch.zeros(len(indices), dtype=F64, device="cuda"),
            "it": (C.c_int64 * S)(), "res": (C.c_double * S)()}


def _level1_inputs(case, seed):
    g = _gen(seed)
    x, r, p, q = (torch.randn(case["n"], generator=g, device="cuda", dtype=F64) for _ in range(4))
    return x, r, p, 2 * p + 0.5 * q     # q = A p of a positive definite A


def _prepare_level1(case, seed):
    x, r, p, q = _level1_inputs(case, seed)

    def bits(v):
        return int(np.float64(v).view(np.uint64))
    steps = (abi.VecStep * 3)()
    # x += alpha p; r += -alpha q; rr += r . r
    for k, (z, y, s) in enumerate(((0, 2, 1e-3), (1, 3, -1e-3))):
        steps[k] = abi.VecStep(kind=abi.VEC_MULADD, op=abi.OP_ADD, mul_op=abi.OP_MUL, z=z, x=-1,
                               y=y, alpha=bits(s))
    steps[2] = abi.VecStep(kind=abi.VEC_REDUCE, op=abi.OP_ADD, mul_op=abi.OP_MUL, z=-1, x=1, y=1)
    vals = (C.c_void_p * 4)(x.data_ptr(), r.data_ptr(), p.data_ptr(), q.data_ptr())
    return {"n": case["n"], "x": x, "r": r, "p": p, "q": q, "steps": steps, "vals": vals,
            "types": (C.c_int * 4)(*[abi.FP64] * 4)}


# -------------------------------------------------------------------- run --
def run(st: dict):
    return globals()["_run_" + st["kind"]](st)


def _run_mxv(st):
    A, u = st["A"], st["u"]
    if "mask" in st:    # a traversal step writes a new sparse vector
        ua, nnz = st["u_assigned"], st["u_nnz"]
        u.zero_()
        ua.zero_()
        nnz.zero_()
        dev.mxv(st["ring"], A, u, st["v"], descr=abi.DESC_INVERT_MASK | abi.DESC_STRUCTURAL,
                u_assigned=ua, u_nnz=nnz, u_mask=st["mask"], u_mask_assigned=st["mask_assigned"],
                u_mask_count=st["mask_count"], v_assigned=st["v_assigned"], v_count=st["v_count"],
                plan=st["plan"])
        return u, ua, nnz
    if "v_assigned" in st:
        dev.mxv(st["ring"], A, u, st["v"], v_assigned=st["v_assigned"], v_count=st["v_count"],
                plan=st["plan"])
        return u
    if u.dtype == torch.uint8:
        u.zero_()       # rows already true would be skipped
    dev.mxv(st["ring"], A, u, st["v"], plan=st["plan"])
    return u


def _run_cg(st):
    A = st["A"]
    st["x"].zero_()
    abi.call("alpb_cg_solve", A.m, *A.p(), dev.ptr(st["b"]), dev.ptr(st["x"]), 2000, 1e-10,
             C.byref(st["iterations"]), C.byref(st["residual"]), dev.ptr(st["work"]),
             st["plan"].h, dev.stream_ptr())
    return st["x"]


def _run_cg_grad(st):
    A, At = st["A"], st["At"]
    abi.call("alpb_cg_grad", A.m, *A.p(), *At.p(), dev.ptr(st["b"]), dev.ptr(st["target"]),
             dev.ptr(st["x"]), dev.ptr(st["lam"]), dev.ptr(st["grad"]), dev.ptr(st["work"]), 5000,
             1e-12, C.byref(st["loss"]), C.byref(st["it"][0]), C.byref(st["it"][1]),
             st["plan"].h, st["plan_t"].h, dev.stream_ptr())
    return {"loss": np.array([st["loss"].value]), "x": st["x"], "dl_db": st["lam"], "dl_da": st["grad"]}


def _run_batched_cg(st):
    st["x"].zero_()
    s, h = dev.stream_ptr(), st["h"].h
    abi.call("alpb_batched_cg_solve", h, dev.ptr(st["b"]), dev.ptr(st["x"]), 20000, 1e-8, s)
    at = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    abi.call("alpb_batched_cg_results", h, at(st["it"]), at(st["rr"]), at(st["conv"]), s)
    return st["x"], st["conv"]


def _run_pagerank(st):
    L, LT = st["L"], st["LT"]
    abi.call("alpb_pagerank_planned", L.m, *L.p(), *LT.p(), dev.ptr(st["pr"]), 0, 0.85, 1e-9, 1000,
             C.byref(st["it"]), C.byref(st["res"]), dev.ptr(st["work"]), st["plan"].h,
             dev.stream_ptr())
    return st["pr"], st["it"].value


def _run_hpcg(st):
    st["x"].zero_()
    abi.call("alpb_hpcg_solve", st["h"].h, dev.ptr(st["b"]), dev.ptr(st["x"]), 1, 1, 1, st["max"],
             1e-30, st["it"], st["res"], dev.stream_ptr())
    return st["x"]      # the residual norm, after ten steps, is all rounding of the first


def _run_ppr(st):
    h, s = st["h"].h, dev.stream_ptr()
    abi.call("alpb_ppr_solve", h, st["seeds"].ctypes.data_as(C.c_void_p), 0.85, 1e-9, 1000,
             dev.ptr(st["x"]), 0, st["it"], st["res"], s)
    abi.call("alpb_ppr_adjoint", h, dev.ptr(st["dl_dx"]), dev.ptr(st["lam"]), 1e-9, 2000, st["it"],
             st["res"], s)
    abi.call("alpb_ppr_grad_weights", h, dev.ptr(st["x"]), dev.ptr(st["lam"]),
             dev.ptr(st["grad"]), s)
    return {"x": st["x"], "lambda": st["lam"], "dl_dw": st["grad"]}


def _run_level1(st):
    n, s = st["n"], dev.stream_ptr()
    pq, rr = C.c_double(0.0), C.c_double(0.0)
    abi.call("alpb_dot_f64", C.byref(pq), abi.OP_ADD, abi.OP_MUL, n, dev.ptr(st["p"]), None,
             dev.ptr(st["q"]), None, s)
    abi.call("alpb_vec_chain", abi.FP64, n, 4, st["vals"], st["types"], 3, st["steps"],
             C.byref(rr), s)
    # p = 0.5 p + r
    abi.call("alpb_foldl_f64", dev.ptr(st["p"]), abi.OP_MUL, n, None, 0.5, s)
    abi.call("alpb_foldl_f64", dev.ptr(st["p"]), abi.OP_ADD, n, dev.ptr(st["r"]), 0.0, s)
    return {"pq": np.array([pq.value]), "rr": np.array([rr.value]), "x": st["x"], "r": st["r"], "p": st["p"]}


# ------------------------------------------------------------------- work --
def _rmat_nnz(m, n, edge_factor):
    # about 3 % of the draws are duplicates at scale 22, 10-20 % on small graphs
    return int(edge_factor * min(m, n) * 0.9)


def work(case: dict) -> dict:
    """Each input read once and each output written once; a solver's operations
    are those of its usual iteration count."""
    k = case["kind"]
    if k == "mxv":
        m, n = case["m"], case["n"]
        nnz = {"rmat": _rmat_nnz(m, n, case.get("edge_factor", 0)), "27pt": 27 * m,
               "5pt": 5 * m}[case["graph"]]
        vb = {"plus_times_f64": 8, "min_plus_i32": 4, "lor_land_bool": 1}[case["ring"]]
        mb = 0 if case["ring"] == "lor_land_bool" else vb
        extra = (n if case["frontier"] else 0) + (2 * m if case["visited"] else 0)
        return {"bytes": nnz * (4 + mb) + 8 * (m + 1) + n * vb + 2 * m * vb + extra,
                "flops": 2 * nnz}
    if k in ("cg", "cg_grad"):
        n = case["nx"] * case["ny"] * case["nz"]
        its = (2.2 * max(case["nx"], case["ny"], case["nz"]) if k == "cg" else 200)
        passes = 1 if k == "cg" else 2
        return {"bytes": passes * (12 * 27 * n + 8 * n + 16 * n) + (8 * 27 * n if k != "cg" else 0),
                "flops": int(its * passes * (54 + 12) * n)}
    if k == "batched_cg":
        lo, hi = case["lo"], case["hi"]
        rows = case["systems"] * (hi * hi - lo * lo) / (2 * math.log(hi / lo))
        return {"bytes": int(rows * (12 * 5 + 8 + 16)), "flops": int(150 * rows * 22)}
    if k == "pagerank":
        nnz = _rmat_nnz(case["n"], case["n"], case["edge_factor"])
        return {"bytes": 12 * nnz + 16 * case["n"] + 8 * case["n"], "flops": 30 * 2 * nnz}
    if k == "hpcg":
        n = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": int((12 * 27 + 8 + 24 * case["nrhs"]) * n * 8 / 7),
                "flops": int(case["iterations"] * 5 * 54 * n * case["nrhs"] * 8 / 7)}
    if k == "ppr":
        nnz, S = _rmat_nnz(case["n"], case["n"], case["edge_factor"]), case["seeds"]
        return {"bytes": 20 * nnz + 16 * S * case["n"] + 8 * S * case["n"],
                "flops": 300 * 2 * nnz * S}
    return {"bytes": (2 + 6 + 2) * 8 * case["n"], "flops": 10 * case["n"]}


def tolerance(case: dict):
    """FP64 sums in another order: measured 1e-16 (stencil rows) to 5.6e-15 (the
    hub rows of a scale-22 graph) from the 64-bit sums.  A solver stops at a
    residual, and one that rounds otherwise may stop one step apart: measured
    from the solution, cg 8e-10, cg_grad 9e-12, batched_cg 2e-8, pagerank
    5e-10, ppr 2.4e-9; after a fixed number of steps, hpcg 6e-16."""
    if case["kind"] == "mxv":
        return {"rel": 2e-14, "max": 1e-12} if case["ring"] == "plus_times_f64" else "exact"
    return {"cg": {"rel": 1e-8}, "cg_grad": {"rel": 1e-10}, "batched_cg": {"rel": 1e-7},
            "pagerank": {"rel": 2e-9}, "hpcg": {"rel": 1e-13}, "ppr": {"rel": 1e-8},
            "level1": {"rel": 1e-13}}[case["kind"]]


# ------------------------------------------------------------------ exact --
def _spmv(offsets, indices, values, x):
    # sequential per row is enough: 64-bit products and sums
    m = len(offsets) - 1
    return torch.zeros(m, dtype=F64, device="cuda").index_add_(
        0, _row_index(offsets), values * x[indices.to(torch.int64)])


def _sparse(offsets, indices, values, n):
    return torch.sparse_csr_tensor(offsets, indices.to(torch.int64), values,
                                   size=(len(offsets) - 1, n))


def _cg_plain(A, b, iterations):
    x, r = torch.zeros_like(b), b.clone()
    p, rr = r.clone(), torch.dot(r, r)
    bb = float(rr)
    for _ in range(iterations):
        q = A @ p
        a = rr / torch.dot(p, q)
        x += a * p
        r -= a * q
        new = torch.dot(r, r)
        if float(new) <= 1e-31 * bb:
            break
        p = r + (new / rr) * p
        rr = new
    return x


def exact(case: dict, seed: int):
    return globals()["_exact_" + case["kind"]](case, seed)


def _exact_mxv(case, seed):
    if case["ring"] != "plus_times_f64":
        return None
    d = _mxv_inputs(case, seed)
    return d["u"] + _spmv(d["offsets"], d["indices"], d["values"], d["v"])


def _exact_cg(case, seed):
    return _cg_inputs(case, seed)[4]


def _exact_cg_grad(case, seed):
    offsets, indices, values, b, target = _cg_grad_inputs(case, seed)
    A = _sparse(offsets, indices, values, len(b))
    x = _cg_plain(A, b, 3000)
    lam = _cg_plain(A, x - target, 3000)    # A is symmetric
    grad = -lam[_row_index(offsets)] * x[indices.to(torch.int64)]
    return {"loss": 0.5 * torch.dot(x - target, x - target).view(1), "x": x, "dl_db": lam,
            "dl_da": grad}


def _exact_batched_cg(case, seed):
    """each 5-point system is diagonal in the sine basis of its two dimensions"""
    sides, shifts, _, _, _, b = _batch_inputs(case, seed)
    out, at = torch.empty_like(b), 0
    for L, shift in zip(sides.tolist(), shifts.tolist()):
        k = torch.arange(1, L + 1, device="cuda", dtype=F64)
        S = torch.sin(math.pi / (L + 1) * k[:, None] * k[None, :]) * math.sqrt(2.0 / (L + 1))
        ev = 2.0 - 2.0 * torch.cos(math.pi / (L + 1) * k)
        B = b[at:at + L * L].view(L, L)
        X = S @ ((S @ B @ S) / (ev[:, None] + ev[None, :] + shift)) @ S
        out[at:at + L * L] = X.reshape(-1)
        at += L * L
    return out, None


def _exact_pagerank(case, seed):
    n = case["n"]
    offsets, indices = _rmat(n, n, case["edge_factor"], _gen(seed))
    deg = (offsets[1:] - offsets[:-1]).to(F64)
    scale = torch.where(deg > 0, 0.85 / deg.clamp(min=1), torch.zeros_like(deg))
    rows, cols = _row_index(offsets), indices.to(torch.int64)
    pr = torch.full((n,), 1.0 / n, dtype=F64, device="cuda")
    for _ in range(250):
        dangling = pr[deg == 0].sum()
        new = torch.zeros_like(pr).index_add_(0, cols, (pr * scale)[rows])
        new += (0.85 * dangling + 0.15) / n
        change = float((new - pr).abs().sum())
        pr = new
        if change <= 1e-15:
            break
    return pr, None


def _exact_hpcg(case, seed):
    dims, nrhs = (case["nx"], case["ny"], case["nz"]), case["nrhs"]
    b = torch.randn(dims[0] * dims[1] * dims[2] * nrhs, generator=_gen(seed), device="cuda",
                    dtype=F64).view(-1, nrhs)
    levels = []
    for _ in range(case["levels"] + 1):
        if levels and min(dims) < 4:
            break
        nx, ny, nz = dims
        n = nx * ny * nz
        i = torch.arange(n, device="cuda")
        x, y, z = i % nx, (i // nx) % ny, i // (nx * ny)
        nb = torch.full((n, 27), n, device="cuda")     # row n stands for "outside": zero
        c = 0
        for dz in (-1, 0, 1):
            for dy in (-1, 0, 1):
                for dx in (-1, 0, 1):
                    ok = ((x + dx >= 0) & (x + dx < nx) & (y + dy >= 0) & (y + dy < ny) &
                          (z + dz >= 0) & (z + dz < nz))
                    nb[:, c] = torch.where(ok, i + dx + nx * (dy + ny * dz), n)
                    c += 1
        cx, cy, cz = nx // 2, ny // 2, nz // 2
        j = torch.arange(cx * cy * cz, device="cuda")
        inj = 2 * (j % cx) + 2 * ((j // cx) % cy) * nx + 2 * (j // (cx * cy)) * nx * ny
        levels.append((n, nb, inj))
        dims = (cx, cy, cz)

    def product(level, v, rows=None):       # v has the extra zero row
        n, nb, _ = levels[level]
        idx = nb if rows is None else nb[rows]
        own = v[:n] if rows is None else v[rows]
        return 27.0 * own - v[idx].sum(1)

    def smooth(level, r, z):
        n = levels[level][0]
        for order in (range(27), range(26, -1, -1)):
            for c in order:
                rows = torch.arange(c, n, 27, device="cuda")
                z[rows] += (r[rows] - product(level, z, rows)) / 26.0

    def cycle(level, r):
        n, _, inj = levels[level]
        z = torch.zeros(n + 1, nrhs, dtype=F64, device="cuda")
        smooth(level, r, z)
        if level + 1 < len(levels):
            coarse = cycle(level + 1, r[inj] - product(level, z, inj))
            z[inj] += coarse[:-1]
            smooth(level, r, z)
        return z

    def pad(v):
        return torch.cat([v, v.new_zeros(1, nrhs)])
    x, r = torch.zeros_like(b), b.clone()
    p, rz = None, None
    for _ in range(case["iterations"]):
        z = cycle(0, r)[:-1]
        new = (r * z).sum(0)
        p = z.clone() if p is None else (new / rz) * p + z
        rz = new
        ap = product(0, pad(p))
        alpha = rz / (p * ap).sum(0)
        x += alpha * p
        r -= alpha * ap
    return x.reshape(-1)


def _exact_ppr(case, seed):
    n, S = case["n"], case["seeds"]
    offsets, indices, weights, seeds, dl_dx = _ppr_inputs(case, seed)
    rows, cols = _row_index(offsets), indices.to(torch.int64)
    deg = torch.zeros(n, dtype=F64, device="cuda").index_add_(0, rows, weights)
    w = 0.85 * weights / deg[rows]
    A = _sparse(offsets, indices, w, n)
    t_off, t_idx, t_val = _transpose(offsets, indices, w, n)
    At = _sparse(t_off, t_idx, t_val, n)
    dang = (deg == 0).to(F64)[:, None]
    sd = torch.from_numpy(np.asarray(seeds)).cuda()
    s = torch.arange(S, device="cuda")
    x = torch.full((n, S), 1.0 / n, dtype=F64, device="cuda")
    g = dl_dx.view(n, S)
    lam = g.clone()
    for _ in range(300):
        mass = 0.85 * (x * dang).sum(0) + 0.15
        x = At @ x
        x[sd, s] += mass
    for _ in range(400):
        lam = A @ lam + 0.85 * dang * lam[sd, s] + g
    mu = (A @ lam) / 0.85
    grad = torch.empty_like(weights)
    for a in range(0, len(rows), 1 << 20):
        i, j = rows[a:a + (1 << 20)], cols[a:a + (1 << 20)]
        grad[a:a + (1 << 20)] = 0.85 / deg[i] * (x[i] * (lam[j] - mu[i])).sum(1)
    return {"x": x.reshape(-1), "lambda": lam.reshape(-1), "dl_dw": grad}


def _exact_level1(case, seed):
    x, r, p, q = _level1_inputs(case, seed)
    pq = torch.dot(p, q).view(1)
    x, r = x + 1e-3 * p, r - 1e-3 * q
    return {"pq": pq, "rr": torch.dot(r, r).view(1), "x": x, "r": r, "p": 0.5 * p + r}
