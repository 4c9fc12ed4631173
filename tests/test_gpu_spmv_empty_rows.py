"""Runs of empty rows in the nonzero-tiled walk (csrc/spmv_merge_path_nz.cuh):
runs around the 256 row ends of a tile and the 32 of a window, before, between
and after rows of every length, with row scales, and matrices of empty rows
alone; equal positions, rows at tile edges."""
import numpy as np
import pytest
import torch

from conftest import order_free_bound

pytestmark = pytest.mark.gpu

WALKS = [("merge_path", {"nz_per_lane": 8}), ("merge_path", {"nz_per_lane": 16}),
         ("merge_path", {"nz_per_lane": 8, "compensated": True}),
         ("merge_path", {"nz_per_lane": 8, "max_ctas": 1}),
         ("work_oriented", {"num_threads": 128}), ("work_oriented", {"num_threads": 4096}),
         ("group_mapped", {}), ("group_mapped", {"group_rows": 32})]


def lengths(name, rng):
    if name == "all empty":
        return np.zeros(5000, np.int64)
    parts = []
    for run in (1, 31, 32, 33, 255, 256, 257, 287, 511, 512, 513, 767, 768, 1024, 2500):
        parts.append(np.zeros(run, np.int64))
        if name == "one by one":
            parts.append(np.ones(1, np.int64))
        elif name == "tiles":  # whole tiles of 256 and 512 nonzeros, and one off
            parts.append(rng.choice([255, 256, 257, 512, 1]) * np.ones(1, np.int64))
        else:
            parts.append(rng.integers(1, 40, rng.integers(1, 30)))
    return np.concatenate(parts if name != "ends full" else parts[1:])


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("name", ["all empty", "one by one", "tiles", "ragged", "ends full"])
def test_runs_of_empty_rows(cuda, oracle_mod, name, dtype):
    from edge_loops_gb300 import api
    rng = np.random.default_rng(len(name))
    lens, cols = lengths(name, rng), 900
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    idx = rng.integers(0, cols, off[-1]).astype(np.int32)
    vals = rng.uniform(-1, 1, off[-1]).astype(np.float32)
    x = rng.uniform(-1, 1, cols).astype(np.float32)
    A = api.CSR.from_arrays(off, idx, vals, cols, device=cuda)
    scale = None
    if dtype != "f32":
        A = A.quantized(torch.bfloat16)
        scale = A.row_scale.cpu().numpy()
    y64, yabs = oracle_mod.spmv_f64(off, idx, A.values.float().cpu().numpy(), x, row_scale=scale)
    xt = torch.as_tensor(x, device=cuda)
    for schedule, opts in WALKS:
        y = torch.full((A.rows,), float("nan"), device=cuda)
        api.spmv(A, xt, y, schedule=schedule, **opts)
        assert api.workspace_errors() == 0
        assert np.all(np.abs(y.cpu().numpy() - y64) <= order_free_bound(off, yabs, extra=3))


def test_many_empty_rows_by_few_threads(cuda):
    """128 threads over 300,000 empty rows: 0.3 ms by a thread per even share,
    3.9 ms when a lane took the ends of a tile one by one (the bound, 1.5 ms,
    stands between)."""
    from edge_loops_gb300 import api
    A = api.CSR(torch.zeros(300_001, dtype=torch.int32, device=cuda),
                torch.empty(0, dtype=torch.int32, device=cuda), torch.empty(0, device=cuda),
                300_000, 100)
    x, y = torch.ones(100, device=cuda), torch.full((300_000,), 3.0, device=cuda)
    best = float("inf")
    for _ in range(6):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        api.spmv(A, x, y, schedule="work_oriented", num_threads=128)
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b))
    assert not bool(y.any()) and best < 1.5
