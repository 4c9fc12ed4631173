"""The work this library is measured on: calls a user's program makes through
the public entry points (edge_loops_gb300.api), over the range of sizes,
shapes and value types they are made with.

Every case is a dict of plain values.  `op` says which entry point:

  spmv     y = A x with one schedule (`merge_path` is the default a caller
           gets; `selected` is what api.select_schedule picks for the matrix,
           asked once, as a solver would)
  spmm     C = A B for a dense row-major B of `n` columns
  batched  one pass of a kept batch plan over `count` matrices
  coo      CSR from unsorted COO entries (a loader's or assembler's output)

and `kind` how the matrix looks: `uniform` (equal rows, scattered columns),
`powerlaw` (Zipf row lengths: graphs), `lognormal` (ragged rows), `stencil`
(27-point stencil on a cube: solvers).
"""
import math

import torch

from edge_loops_gb300 import api, synth

_DT = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
_DEV = "cuda"


def listed():
    return [
        # the smallest call: one short SpMV, where launch and host time count
        {"name": "spmv_uniform1k_f32", "op": "spmv", "kind": "uniform", "rows": 1000, "cols": 1000,
         "mean": 10, "dtype": "f32", "schedule": "merge_path"},
        # a graph's adjacency matrix (PageRank-like iteration), default schedule
        {"name": "spmv_powerlaw16m_f32", "op": "spmv", "kind": "powerlaw", "rows": 1 << 20,
         "cols": 1 << 20, "mean": 15, "dtype": "f32", "schedule": "merge_path"},
        # a rectangular ragged matrix of odd sizes with 16-bit values and row scales
        {"name": "spmv_lognormal4m_f16", "op": "spmv", "kind": "lognormal", "rows": 300007,
         "cols": 251111, "mean": 13, "dtype": "f16", "schedule": "merge_path"},
        # one matrix-vector product of an iterative solver on a 3-D grid, by
        # a caller who asks for nothing but the default
        {"name": "spmv_stencil160_f32", "op": "spmv", "kind": "stencil", "grid": 160,
         "dtype": "f32", "schedule": "merge_path"},
        # the same solver, 16-bit matrix, with the schedule the library picks
        {"name": "spmv_stencil128_bf16_selected", "op": "spmv", "kind": "stencil", "grid": 128,
         "dtype": "bf16", "schedule": "selected"},
        # the reference's other schedules, by callers who name them
        {"name": "spmv_work_oriented16m_f32", "op": "spmv", "kind": "lognormal", "rows": 2000003,
         "cols": 2000003, "mean": 8, "dtype": "f32", "schedule": "work_oriented"},
        {"name": "spmv_group_mapped_stencil96_f32", "op": "spmv", "kind": "stencil", "grid": 96,
         "dtype": "f32", "schedule": "group_mapped"},
        # many independent small systems in one launch
        {"name": "batched1024_bf16", "op": "batched", "count": 1024, "rows_lo": 64,
         "rows_hi": 65536, "mean": 8, "dtype": "bf16"},
        # graph features: adjacency matrix times a narrow and a wide dense matrix
        {"name": "spmm_powerlaw8m_n32_f32", "op": "spmm", "kind": "powerlaw", "rows": 1 << 20,
         "cols": 1 << 20, "mean": 7.6, "dtype": "f32", "n": 32, "b_dtype": "f32",
         "schedule": "merge_path"},
        {"name": "spmm_powerlaw8m_n128_bf16", "op": "spmm", "kind": "powerlaw", "rows": 1 << 20,
         "cols": 1 << 20, "mean": 7.6, "dtype": "f32", "n": 128, "b_dtype": "bf16",
         "schedule": "merge_path"},
        # the reference's own SpMM schedule (row order kept), odd sizes
        {"name": "spmm_thread_mapped2m_n24_f32", "op": "spmm", "kind": "lognormal", "rows": 200003,
         "cols": 150001, "mean": 10, "dtype": "f32", "n": 24, "b_dtype": "f32",
         "schedule": "thread_mapped"},
        # building the graph's CSR from its shuffled edge list
        {"name": "coo_powerlaw16m", "op": "coo", "kind": "powerlaw", "rows": 1 << 20,
         "cols": 1 << 20, "mean": 15},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _matrix(rng, kinds, nnz_lo, nnz_hi):
    """A matrix of one of `kinds` with about nnz_lo .. nnz_hi nonzeros."""
    kind = rng.choice(kinds)
    nnz = _log_int(rng, nnz_lo, nnz_hi)
    if kind == "stencil":
        n = max(8, min(160, round((nnz ** (1 / 3) + 2) / 3)))
        return {"kind": kind, "grid": max(8, min(160, n + rng.choice([-1, 0, 1])))}
    mean = rng.randint(3, 40) if kind != "powerlaw" else rng.randint(4, 20)
    rows = max(200, min(4_000_000, nnz // mean)) + rng.randint(0, 63)
    cols = max(200, min(4_000_000, int(rows * rng.uniform(0.5, 2.0)))) + rng.randint(0, 63)
    return {"kind": kind, "rows": rows, "cols": cols, "mean": mean}


def draw(rng):
    op = rng.choice(["spmv", "spmv", "spmv", "spmm", "spmm", "batched", "coo"])
    if op == "spmv":
        schedule = rng.choice(["merge_path", "merge_path", "merge_path", "selected",
                               "work_oriented", "group_mapped"])
        kinds = ["uniform", "lognormal", "stencil"]
        if schedule in ("merge_path", "selected"):
            kinds.append("powerlaw")
        hi = 30_000_000 if schedule in ("merge_path", "selected") else 16_000_000
        m = _matrix(rng, kinds, 6_000, hi)
        return dict(m, op=op, schedule=schedule, dtype=rng.choice(["f32", "f32", "bf16", "f16"]))
    if op == "spmm":
        schedule = rng.choice(["merge_path", "merge_path", "merge_path", "thread_mapped",
                               "group_mapped"])
        if schedule == "merge_path":
            m = _matrix(rng, ["uniform", "lognormal", "stencil", "powerlaw"], 20_000, 8_000_000)
            n = _log_int(rng, 2, 160)
        else:
            m = _matrix(rng, ["uniform", "lognormal", "stencil"], 20_000, 2_000_000)
            n = _log_int(rng, 2, 64)
        dtype = rng.choice(["f32", "f32", "bf16"])
        return dict(m, op=op, schedule=schedule, dtype=dtype, n=n,
                    b_dtype=rng.choice(["f32", "bf16"]))
    if op == "batched":
        lo = _log_int(rng, 64, 1000)
        hi, mean = lo + _log_int(rng, 1000, 64000), rng.randint(4, 16)
        most = 75_000_000 * math.log(hi / lo) / ((hi - lo) * mean)  # nonzeros in all
        return {"op": op, "count": min(_log_int(rng, 8, 1000), int(most)), "rows_lo": lo,
                "rows_hi": hi, "mean": mean, "dtype": rng.choice(["f32", "bf16", "f16"])}
    return dict(_matrix(rng, ["uniform", "lognormal", "powerlaw"], 20_000, 15_000_000), op=op)


# ------------------------------------------------------------------- inputs
def _csr_arrays(case, seed):
    """offsets, indices, values (f32), x, rows, cols of the case's matrix."""
    kind = case["kind"]
    if kind == "stencil":
        off, idx, val, x, n = synth.stencil27(case["grid"], seed=seed, device=_DEV)
        return off, idx, val, x, n, n
    rows, cols = case["rows"], case["cols"]
    if kind == "uniform":
        off, idx, val, x, _ = synth.uniform_rows(rows, cols, case["mean"], seed=seed, device=_DEV)
        return off, idx, val, x, rows, cols
    # ragged rows: the lengths are the case's own (the same multiset for every
    # seed, so that the sizes are too), which row has which, the columns, the
    # values and x are the seed's
    g = torch.Generator(device=_DEV)
    g.manual_seed(1)
    if kind == "powerlaw":  # Zipf(2) on [1, 100000], scaled to the mean
        cap = min(100_000, cols)
        cdf = torch.cumsum(torch.arange(1, cap + 1, device=_DEV, dtype=torch.float64).pow(-2.0), 0)
        u = torch.rand(rows, generator=g, device=_DEV, dtype=torch.float64) * cdf[-1]
        lens = torch.searchsorted(cdf, u).clamp_(max=cap - 1).double() + 1.0
        lens = torch.round(lens * (case["mean"] * rows / lens.sum())).clamp_(1, cap)
    else:  # log-normal, sigma 1; some rows are empty
        z = torch.randn(rows, generator=g, device=_DEV, dtype=torch.float64)
        lens = torch.round(torch.exp(math.log(case["mean"]) - 0.5 + z)).clamp_(max=cols)
    g.manual_seed(int(seed))
    lens = lens.long()[torch.randperm(rows, generator=g, device=_DEV)]
    off = torch.zeros(rows + 1, dtype=torch.int64, device=_DEV)
    off[1:] = torch.cumsum(lens, 0)
    nnz = int(off[-1])
    # columns uniform and sorted within the row (one may repeat, as in an
    # assembly that is not summed yet)
    row_of = torch.repeat_interleave(torch.arange(rows, device=_DEV), lens)
    col = torch.randint(0, cols, (nnz,), generator=g, device=_DEV)
    key, _ = torch.sort(row_of * cols + col)
    idx = (key - row_of * cols).to(torch.int32)
    val = torch.rand(nnz, generator=g, device=_DEV) * 2 - 1
    x = torch.rand(cols, generator=g, device=_DEV) * 2 - 1
    return off.to(torch.int32), idx, val, x, rows, cols


def _matrix_and_x(case, seed):
    off, idx, val, x, rows, cols = _csr_arrays(case, seed)
    A = api.CSR(off, idx, val, rows, cols)
    if case["dtype"] != "f32":
        A = A.quantized(_DT[case["dtype"]])
    return A, x


def _batch(case, seed):
    # the matrices' pattern is the case's own, the values and x the seed's
    rows, off, idx, val, x, row_start, nz_start = synth.batched(
        case["count"], case["rows_lo"], case["rows_hi"], case["mean"], device=_DEV)
    g = torch.Generator(device=_DEV)
    g.manual_seed(int(seed))
    val = torch.rand(val.numel(), generator=g, device=_DEV) * 2 - 1
    x = torch.rand(x.numel(), generator=g, device=_DEV) * 2 - 1
    items, y = api.batched_items(rows, off, idx, val, x, row_start, nz_start)
    if case["dtype"] != "f32":
        # one values array and one scales array, at the offsets of the indices
        v16 = torch.empty(idx.numel(), dtype=_DT[case["dtype"]], device=_DEV)
        sc = torch.empty(x.numel(), dtype=torch.float32, device=_DEV)
        rs, ns = row_start.tolist(), nz_start.tolist()
        items = [(A.quantized(_DT[case["dtype"]], out=v16[ns[m]: ns[m] + A.nnz],
                              out_scale=sc[rs[m]: rs[m] + A.rows]), xm, ym)
                 for m, (A, xm, ym) in enumerate(items)]
    return items, x, y


def _dense(case, seed, cols):
    g = torch.Generator(device=_DEV)
    g.manual_seed(int(seed) + 7919)
    B = torch.rand(cols, case["n"], generator=g, device=_DEV) * 2 - 1
    return B.to(_DT[case["b_dtype"]])


def _coo(case, seed):
    off, idx, val, _, rows, cols = _csr_arrays(case, seed)
    g = torch.Generator(device=_DEV)
    g.manual_seed(int(seed) + 104729)
    row_of = torch.repeat_interleave(torch.arange(rows, device=_DEV, dtype=torch.int32),
                                     (off[1:] - off[:-1]).long())
    p = torch.randperm(idx.numel(), generator=g, device=_DEV)
    return rows, cols, row_of[p], idx[p], val[p]


def prepare(case, seed):
    op = case["op"]
    if op == "coo":
        return {"case": case, "coo": _coo(case, seed)}
    if op == "batched":
        items, _, y = _batch(case, seed)
        return {"case": case, "plan": api.BatchPlan(items), "y": y}
    A, x = _matrix_and_x(case, seed)
    if op == "spmm":
        C = torch.empty(A.rows, case["n"], dtype=torch.float32, device=_DEV)
        return {"case": case, "A": A, "B": _dense(case, seed, A.cols), "C": C}
    schedule, opts = case["schedule"], {}
    if schedule == "selected":
        schedule, opts = api.select_schedule(A)
    y = torch.empty(A.rows, dtype=torch.float32, device=_DEV)
    return {"case": case, "A": A, "x": x, "y": y, "schedule": schedule, "opts": opts}


def run(state):
    op = state["case"]["op"]
    if op == "spmv":
        return api.spmv(state["A"], state["x"], state["y"], schedule=state["schedule"],
                        **state["opts"])
    if op == "spmm":
        return api.spmm(state["A"], state["B"], state["C"], schedule=state["case"]["schedule"])
    if op == "batched":
        state["plan"].execute()
        return state["y"]
    A = api.csr_from_coo(*state["coo"])
    return A.offsets, A.indices, A.values


# --------------------------------------------------------------------- work
def _sizes(case):
    """rows, cols, nonzeros (expected) of the case's matrix."""
    if case["kind"] == "stencil":
        n = case["grid"]
        return n ** 3, n ** 3, (3 * n - 2) ** 3
    return case["rows"], case["cols"], int(case["rows"] * case["mean"])


def work(case):
    if case["op"] == "batched":
        lo, hi = math.log(case["rows_lo"]), math.log(case["rows_hi"])
        rows = case["count"] * (case["rows_hi"] - case["rows_lo"]) / (hi - lo)
        cols, nnz = rows, rows * case["mean"]
    else:
        rows, cols, nnz = _sizes(case)
    if case["op"] == "coo":
        return {"bytes": nnz * 12 + 4 * (rows + 1) + nnz * 8, "flops": 0}
    vb = 4 if case["dtype"] == "f32" else 2
    matrix = nnz * (4 + vb) + 4 * (rows + 1) + (0 if vb == 4 else 4 * rows)
    if case["op"] == "spmm":
        n, bb = case["n"], 4 if case["b_dtype"] == "f32" else 2
        return {"bytes": matrix + cols * n * bb + 4 * rows * n, "flops": 2 * nnz * n}
    return {"bytes": matrix + 4 * cols + 4 * rows, "flops": 2 * nnz}


# -------------------------------------------------------------------- exact
def _rows_of(off):
    rows = off.numel() - 1
    return torch.repeat_interleave(torch.arange(rows, device=off.device),
                                   (off[1:] - off[:-1]).long())


def _dequantized(A):
    v = A.values[: A.nnz].double()
    return v if A.row_scale is None else v * A.row_scale.double()[_rows_of(A.offsets)]


def exact(case, seed):
    op = case["op"]
    if op == "coo":
        rows, cols, ri, ci, val = _coo(case, seed)
        key, order = torch.sort(ri.long() * cols + ci.long(), stable=True)
        counts = torch.bincount(ri.long(), minlength=rows)
        off = torch.zeros(rows + 1, dtype=torch.int64, device=_DEV)
        off[1:] = torch.cumsum(counts, 0)
        return off.to(torch.int32), (key % cols).to(torch.int32), val[order].double()
    if op == "batched":
        items, x, y = _batch(case, seed)
        out = torch.zeros(y.numel(), dtype=torch.float64, device=_DEV)
        at = 0
        for A, xm, _ in items:
            p = _dequantized(A) * xm.double()[A.indices.long()]
            out[at: at + A.rows].index_add_(0, _rows_of(A.offsets), p)
            at += A.rows
        return out
    A, x = _matrix_and_x(case, seed)
    v, row_of, col = _dequantized(A), _rows_of(A.offsets), A.indices.long()
    if op == "spmv":
        out = torch.zeros(A.rows, dtype=torch.float64, device=_DEV)
        out.index_add_(0, row_of, v * x.double()[col])
        return out
    B = _dense(case, seed, A.cols)
    out = torch.zeros(A.rows, case["n"], dtype=torch.float64, device=_DEV)
    for c in range(0, case["n"], 8):
        b = B[:, c: c + 8].double()
        out[:, c: c + 8] = torch.zeros(A.rows, b.shape[1], dtype=torch.float64, device=_DEV) \
            .index_add_(0, row_of, v[:, None] * b[col])
    return out
