"""The ordered SpMM on either side of the line between a warp per row and the
walk (csrc/spmm_impl.cuh, few_rows: 5 rows per resident warp, 24 of which are on
an SM; 3 where a lane holds 8 columns): every column layout and type, rows
around the nonzeros in flight, empty rows, rows of thousands.  Both schedules
equal the reference loop bit for bit on both sides."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def matrix(rows, rng):
    lens = rng.integers(0, 5, rows)
    at = rng.choice(rows, 400, replace=False)
    lens[at[:380]] = rng.choice([7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 257], 380)
    lens[at[380:]] = rng.integers(500, 5000, 20)
    lens[[0, rows - 1]] = [300, 33]
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    idx = rng.integers(0, 3000, off[-1]).astype(np.int32)
    return off, idx, rng.uniform(-1, 1, off[-1]).astype(np.float32)


@pytest.mark.parametrize("bdt", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("n", [1, 6, 7, 8, 12, 16, 17, 24, 33, 40, 64, 66, 97, 128, 130])
@pytest.mark.parametrize("per_warp", [3, 5])
def test_both_sides_of_the_line(cuda, oracle_mod, per_warp, n, bdt):
    from edge_loops_gb300 import api
    edge = torch.cuda.get_device_properties(0).multi_processor_count * 24 * per_warp
    dt = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}[bdt]
    rng = np.random.default_rng(n)
    B = torch.as_tensor(rng.uniform(-1, 1, (3000, n)).astype(np.float32), device=cuda).to(dt)
    for rows in (edge, edge + 1):
        off, idx, vals = matrix(rows, rng)
        A = api.CSR.from_arrays(off, idx, vals, 3000, device=cuda)
        exp = oracle_mod.spmm_f32(off, idx, vals, B.float().cpu().numpy())
        for schedule in ("thread_mapped", "group_mapped"):
            C = torch.full((rows, n), float("nan"), device=cuda)
            api.spmm(A, B, C, schedule=schedule)
            assert api.workspace_errors() == 0
            np.testing.assert_array_equal(C.cpu().numpy(), exp)


@pytest.mark.parametrize("rows", [1, 2, 31, 700])
@pytest.mark.parametrize("vdt", ["bf16", "f16"])
def test_few_rows_with_row_scales_and_bad_columns(cuda, oracle_mod, vdt, rows):
    from edge_loops_gb300 import _lib, api
    rng = np.random.default_rng(rows)
    lens = rng.integers(0, 60, rows)
    lens[0] = 45
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    idx = rng.integers(0, 500, off[-1]).astype(np.int32)
    vals = rng.uniform(-1, 1, off[-1]).astype(np.float32)
    dt = torch.bfloat16 if vdt == "bf16" else torch.float16
    for n in (6, 16, 40):
        B = torch.as_tensor(rng.uniform(-1, 1, (500, n)).astype(np.float32), device=cuda)
        A = api.CSR.from_arrays(off, idx, vals, 500, device=cuda).quantized(dt)
        scale = A.row_scale.cpu().numpy()[:, None]  # powers of two: exact
        stored = A.values.float().cpu().numpy()
        C = api.spmm(A, B, schedule="group_mapped")
        assert api.workspace_errors() == 0
        np.testing.assert_array_equal(
            C.cpu().numpy(), oracle_mod.spmm_f32(off, idx, stored, B.cpu().numpy()) * scale)
        A.indices[[0, 40]] = torch.as_tensor([-1, 500], dtype=torch.int32, device=cuda)
        stored[[0, 40]] = 0
        C = api.spmm(A, B, schedule="group_mapped")
        assert api.workspace_errors() == _lib.EL_FLAG_INDEX_RANGE
        np.testing.assert_array_equal(
            C.cpu().numpy(), oracle_mod.spmm_f32(off, idx, stored, B.cpu().numpy()) * scale)
