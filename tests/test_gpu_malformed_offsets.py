"""Malformed offsets: no kernel reads or writes outside the arrays of the CSR,
x, B, y and C.  The indices lie between guards of columns outside [0, cols),
so a read of either guard raises EL_FLAG_INDEX_RANGE; y and C lie between
guards that have to stay as they are.  tests/test_split_bounds.py shows on the
CPU that every access stays inside."""
import numpy as np
import pytest
import torch

from test_split_bounds import offsets

pytestmark = pytest.mark.gpu

GUARD = 4096  # elements on either side
KINDS = ["negative", "first row", "too large", "falls", "reversed", "halves", "random",
         "all negative", "short"]
COLS = 700


def guarded(t, fill, cuda):
    buf = torch.full((t.numel() + 2 * GUARD,), fill, dtype=t.dtype, device=cuda)
    view = buf[GUARD: GUARD + t.numel()]
    view.copy_(t)
    return buf, view


def matrix(kind, rows, rng, cuda):
    """The malformed matrix and a well-formed one of the same indices."""
    from edge_loops_gb300 import api
    good = np.concatenate([[0], np.cumsum(rng.integers(0, 9, rows))]).astype(np.int64)
    off, nnz = (good, int(good[-1])) if kind is None else offsets(kind, rng, rows)
    _, idx = guarded(torch.as_tensor(rng.integers(0, COLS, nnz).astype(np.int32)), COLS, cuda)
    _, vals = guarded(torch.as_tensor(rng.uniform(-1, 1, nnz).astype(np.float32)), float("nan"), cuda)
    return api.CSR(torch.as_tensor(off.astype(np.int32), device=cuda), idx, vals, rows, COLS)


def check(call, ws, width, kind, rows, rng, cuda):
    """call(A, out) on the malformed matrix, then on a well-formed one."""
    from edge_loops_gb300 import _lib
    for k in (kind, None):
        A = matrix(k, rows, rng, cuda)
        buf, out = guarded(torch.zeros(rows * width), 7.5, cuda)
        call(A, out)
        torch.cuda.synchronize()
        flags = ws.errors()
        assert not flags & _lib.EL_FLAG_INDEX_RANGE
        assert bool((buf[:GUARD] == 7.5).all()) and bool((buf[GUARD + rows * width:] == 7.5).all())
    assert flags == 0
    return A, out


@pytest.mark.parametrize("schedule,opts", [
    ("merge_path", {}), ("merge_path", {"nz_per_lane": 8}), ("merge_path", {"nz_per_lane": 16}),
    ("merge_path", {"compensated": True}), ("work_oriented", {}),
    ("work_oriented", {"num_threads": 512}), ("work_oriented", {"num_threads": 128 * 304}),
    ("group_mapped", {}), ("group_mapped", {"group_rows": 32})],
    ids=lambda v: v if isinstance(v, str) else "-".join(f"{k}{x}" for k, x in v.items()) or "default")
@pytest.mark.parametrize("rows", [300, 6000])
def test_spmv_stays_inside(cuda, oracle_mod, rows, schedule, opts):
    from edge_loops_gb300 import api
    rng = np.random.default_rng(rows)
    ws = api.Workspace()
    x = torch.as_tensor(rng.uniform(-1, 1, COLS).astype(np.float32), device=cuda)
    for kind in KINDS:
        A, y = check(lambda A, y: api.spmv(A, x, y, schedule=schedule, workspace=ws,
                                           wait_limit_us=2000, **opts),
                     ws, 1, kind, rows, rng, cuda)
        y64, yabs = oracle_mod.spmv_f64(A.offsets.cpu().numpy(), A.indices.cpu().numpy(),
                                        A.values.cpu().numpy(), x.cpu().numpy())
        assert np.all(np.abs(y.cpu().numpy() - y64) <= 12 * 2.0 ** -24 * yabs)


@pytest.mark.parametrize("schedule", ["merge_path", "thread_mapped", "group_mapped"])
@pytest.mark.parametrize("n,bdt", [(4, "f32"), (8, "f32"), (24, "f32"), (32, "bf16"), (128, "f32")])
@pytest.mark.parametrize("rows", [300, 6000, 60_000])
def test_spmm_stays_inside(cuda, oracle_mod, rows, n, bdt, schedule):
    """60,000 rows: the two split points of a block lie up to thousands of rows
    apart where the offsets are not monotone."""
    from edge_loops_gb300 import api
    rng = np.random.default_rng(rows + n)
    ws = api.Workspace()
    B = torch.as_tensor(rng.uniform(-1, 1, (COLS, n)).astype(np.float32), device=cuda)
    B = B.to(torch.bfloat16) if bdt == "bf16" else B
    for kind in KINDS:
        A, C = check(lambda A, C: api.spmm(A, B, C.view(rows, n), schedule=schedule, workspace=ws,
                                           wait_limit_us=2000),
                     ws, n, kind, rows, rng, cuda)
    off, idx, vals = (t.cpu().numpy() for t in (A.offsets, A.indices, A.values))
    got, Bf = C.view(rows, n).cpu().numpy(), B.float().cpu().numpy()
    if schedule == "merge_path":
        C64, Ca = oracle_mod.spmm_f64(off, idx, vals, Bf)
        assert np.all(np.abs(got - C64) <= 12 * 2.0 ** -24 * Ca)
    else:
        np.testing.assert_array_equal(got, oracle_mod.spmm_f32(off, idx, vals, Bf))


@pytest.mark.parametrize("schedule", ["merge_path", "thread_mapped", "group_mapped"])
@pytest.mark.parametrize("kind", ["negative", "too large", "random"])
def test_spmm_flags_bad_offsets(cuda, kind, schedule):
    from edge_loops_gb300 import _lib, api
    rng = np.random.default_rng(11)
    ws = api.Workspace()
    A = matrix(kind, 6000, rng, cuda)
    api.spmm(A, torch.rand(COLS, 24, device=cuda), schedule=schedule, workspace=ws,
             wait_limit_us=2000)
    torch.cuda.synchronize()
    assert ws.errors() & _lib.EL_FLAG_OFFSETS


@pytest.mark.parametrize("kind", ["negative", "int min", "too large", "int max", "falls", "reversed",
                                  "random"])
@pytest.mark.parametrize("schedule,opts", [
    ("merge_path", {}), ("merge_path", {"nz_per_lane": 8}), ("merge_path", {"nz_per_lane": 16}),
    ("work_oriented", {"num_threads": 512}), ("work_oriented", {"num_threads": 128 * 304}),
    ("group_mapped", {}), ("group_mapped", {"group_rows": 32})],
    ids=lambda v: v if isinstance(v, str) else "-".join(f"{k}{x}" for k, x in v.items()) or "default")
def test_spmv_flags_bad_offsets(cuda, kind, schedule, opts):
    """An offset that falls or leaves [0, nnz], wherever it is."""
    from edge_loops_gb300 import _lib, api
    ws = api.Workspace()
    x = torch.rand(COLS, device=cuda)
    for seed in range(12):
        A = matrix(kind, 6000, np.random.default_rng(seed), cuda)
        api.spmv(A, x, schedule=schedule, workspace=ws, wait_limit_us=2000, **opts)
        torch.cuda.synchronize()
        assert ws.errors() & _lib.EL_FLAG_OFFSETS, seed
