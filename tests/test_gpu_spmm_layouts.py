"""The SpMM kernel's layouts and cuts: every column width around the group
sizes (4, 8, 16, 32 lanes of 1, 2, 4 or 8 columns), B and C rows on and off
the vector boundaries, empty rows, rows longer than a block of the walk
(8192 nonzeros), values with row scales, and a malformed CSR.

The ordered schedules equal the reference loop bit for bit
(algorithms/spmm/thread_mapped.cuh:41-52, restated in oracle.c); merge_path
is held to the order-free FP32 bound gamma_(n+2) * sum|a b| (a fused
multiply-add rounds once where the bound counts two)."""
import numpy as np
import pytest
import torch

from conftest import random_csr

pytestmark = pytest.mark.gpu

U = 2.0 ** -24


def strided(rows, n, pad, shift, dtype, cuda):
    """A rows x n view with row stride n + pad whose first element lies
    `shift` elements past an allocation's start (256-byte aligned)."""
    flat = torch.zeros(rows * (n + pad) + shift + 16, dtype=dtype, device=cuda)
    return torch.as_strided(flat, (rows, n), (n + pad, 1), shift)


@pytest.fixture(scope="module")
def ragged():
    rng = np.random.default_rng(5)
    long_rows = [(0, 9000), (3, 12_000), (400, 8192), (401, 8193), (699, 3000)]
    return random_csr(rng, rows=700, cols=20_000, max_len=14, empty_frac=0.3,
                      long_rows=long_rows)[:3]


def as_f32(B):
    return B.float().cpu().numpy()


@pytest.mark.parametrize("bdt", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("n,pad,shift", [
    (1, 0, 0), (2, 0, 0), (3, 1, 1), (4, 0, 0), (5, 3, 0), (8, 0, 0), (9, 0, 0), (12, 0, 0),
    (16, 0, 0), (16, 0, 1), (17, 0, 0), (24, 0, 0), (24, 4, 4), (31, 0, 0), (32, 0, 0),
    (33, 0, 0), (40, 0, 0), (50, 0, 0), (64, 0, 0), (65, 0, 0), (66, 2, 2), (96, 0, 0),
    (97, 0, 0), (100, 0, 0), (128, 0, 0), (128, 1, 0), (129, 0, 0), (160, 0, 0), (257, 0, 0)])
def test_widths_and_alignments(cuda, oracle_mod, ragged, n, pad, shift, bdt):
    from edge_loops_gb300 import api
    off, idx, vals = ragged
    rng = np.random.default_rng(n)
    dt = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}[bdt]
    B = strided(20_000, n, pad, shift, dt, cuda)
    B.copy_(torch.as_tensor(rng.uniform(-1, 1, size=(20_000, n)).astype(np.float32)))
    A = api.CSR.from_arrays(off, idx, vals, 20_000, device=cuda)
    exp = oracle_mod.spmm_f32(off, idx, vals, as_f32(B))
    C64, Ca = oracle_mod.spmm_f64(off, idx, vals, as_f32(B))
    k = (np.diff(off.astype(np.int64)) + 2)[:, None]
    for sched in ("thread_mapped", "group_mapped", "merge_path_flat"):
        C = strided(700, n, pad, shift, torch.float32, cuda)
        C.fill_(float("nan"))
        api.spmm(A, B, C, schedule=sched)
        assert api.workspace_errors() == 0
        got = C.cpu().numpy()
        if sched == "merge_path_flat":
            assert np.all(np.abs(got - C64) <= k * U / (1 - k * U) * Ca)
        else:
            np.testing.assert_array_equal(got, exp)


@pytest.mark.parametrize("vdt,bdt", [("bf16", "bf16"), ("bf16", "f32"), ("f16", "f16"),
                                     ("f16", "f32")])
@pytest.mark.parametrize("n", [3, 16, 24, 33, 128])
@pytest.mark.parametrize("skip", [0, 1])
def test_16bit_values_with_row_scales(cuda, oracle_mod, ragged, n, vdt, bdt, skip):
    """`skip` = 1: the values start 2 bytes off a 4-byte boundary."""
    from edge_loops_gb300 import api
    off, idx, vals = ragged
    dts = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
    rng = np.random.default_rng(n)
    A = api.CSR.from_arrays(off, idx, vals, 20_000, device=cuda)
    store = torch.empty(A.nnz + 1, dtype=dts[vdt], device=cuda)
    A = A.quantized(dts[vdt], out=store[skip: skip + A.nnz])
    B = torch.as_tensor(rng.uniform(-1, 1, size=(20_000, n)).astype(np.float32),
                        device=cuda).to(dts[bdt])
    C64, Ca = oracle_mod.spmm_f64(off, idx, A.values.float().cpu().numpy(), as_f32(B),
                                  row_scale=A.row_scale.cpu().numpy())
    k = (np.diff(off.astype(np.int64)) + 3)[:, None]
    for sched in ("thread_mapped", "merge_path_flat"):
        C = torch.full((700, n), float("nan"), device=cuda)
        api.spmm(A, B, C, schedule=sched)
        assert api.workspace_errors() == 0
        assert np.all(np.abs(C.cpu().numpy() - C64) <= k * U / (1 - k * U) * Ca)


@pytest.mark.parametrize("empty", [0.0, 0.9, 1.0])
def test_many_rows_and_mostly_empty_ones(cuda, oracle_mod, empty):
    """Enough rows for several ranges per warp block, with runs of empty rows
    longer than a window of 32."""
    from edge_loops_gb300 import api
    rng = np.random.default_rng(9)
    rows, cols, n = 60_000, 500, 20
    lens = rng.integers(0, 9, size=rows)
    lens[rng.random(rows) < empty] = 0
    lens[20_000:20_400] = 0
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    idx = rng.integers(0, cols, size=off[-1]).astype(np.int32)
    vals = rng.uniform(-1, 1, size=off[-1]).astype(np.float32)
    B = rng.uniform(-1, 1, size=(cols, n)).astype(np.float32)
    A = api.CSR.from_arrays(off, idx, vals, cols, device=cuda)
    exp = oracle_mod.spmm_f32(off, idx, vals, B)
    C64, Ca = oracle_mod.spmm_f64(off, idx, vals, B)
    for sched in ("group_mapped", "merge_path_flat"):
        C = torch.full((rows, n), float("nan"), device=cuda)
        api.spmm(A, torch.as_tensor(B, device=cuda), C, schedule=sched)
        assert api.workspace_errors() == 0
        got = C.cpu().numpy()
        if sched == "group_mapped":
            np.testing.assert_array_equal(got, exp)
        else:
            k = (lens + 2)[:, None]
            assert np.all(np.abs(got - C64) <= k * U / (1 - k * U) * Ca)


@pytest.mark.parametrize("n", [3, 8, 16, 24, 33, 64, 128])
def test_rows_around_the_long_row_threshold(cuda, oracle_mod, n):
    """Rows of 255 .. 258 nonzeros beside short and empty ones, first, last and
    next to each other: the ordered schedules set the long ones apart."""
    from edge_loops_gb300 import api
    rng = np.random.default_rng(n)
    long_rows = [(0, 257), (1, 256), (2, 258), (3, 257), (40, 255), (41, 0), (42, 600),
                 (43, 0), (100, 4096), (101, 4000), (150, 4097), (151, 4000), (299, 300)]
    off, idx, vals = random_csr(rng, rows=300, cols=6000, max_len=20, empty_frac=0.1,
                                long_rows=long_rows)[:3]
    B = rng.uniform(-1, 1, size=(6000, n)).astype(np.float32)
    A = api.CSR.from_arrays(off, idx, vals, 6000, device=cuda)
    exp = oracle_mod.spmm_f32(off, idx, vals, B)
    for sched in ("thread_mapped", "group_mapped"):
        C = torch.full((300, n), float("nan"), device=cuda)
        api.spmm(A, torch.as_tensor(B, device=cuda), C, schedule=sched)
        assert api.workspace_errors() == 0
        np.testing.assert_array_equal(C.cpu().numpy(), exp)


@pytest.mark.parametrize("sched", ["thread_mapped", "merge_path_flat"])
def test_bad_columns_are_flagged_and_read_nothing(cuda, ragged, sched):
    """Columns outside [0, cols) contribute nothing, whatever B holds, and
    raise the flag (the kernel checks every column before it reads B)."""
    from edge_loops_gb300 import _lib, api
    off, idx, vals = ragged
    bad = idx.copy()
    bad[[5, 9001, 20_000]] = [-1, 20_000, 2 ** 31 - 1]
    keep = np.ones(len(idx), dtype=bool)
    keep[[5, 9001, 20_000]] = False
    for n in (24, 33):
        B = torch.ones(20_000, n, device=cuda)
        C = api.spmm(api.CSR.from_arrays(off, bad, vals, 20_000, device=cuda), B, schedule=sched)
        assert api.workspace_errors() == _lib.EL_FLAG_INDEX_RANGE
        v0 = np.where(keep, vals, 0).astype(np.float32)
        ref = api.spmm(api.CSR.from_arrays(off, idx, v0, 20_000, device=cuda), B, schedule=sched)
        assert api.workspace_errors() == 0
        assert torch.equal(C, ref)


def test_keeps_a_captured_spmv(cuda, ragged):
    """An SpMM takes no more carry slots than a new workspace has, so a graph
    captured with the workspace before it still finds its memory there."""
    from edge_loops_gb300 import api
    off, idx, vals = ragged
    A = api.CSR.from_arrays(off, idx, vals, 20_000, device=cuda)
    x = torch.rand(20_000, device=cuda)
    exp = api.spmv(A, x).cpu()
    y = torch.full((700,), float("nan"), device=cuda)
    ws = api.Workspace()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        api.spmv(A, x, y, workspace=ws)
    C = api.spmm(A, torch.rand(20_000, 8, device=cuda), workspace=ws)
    g.replay()
    torch.cuda.synchronize()
    assert ws.errors() == 0 and torch.equal(y.cpu(), exp) and bool(C.isfinite().all())


@pytest.mark.parametrize("vdt,bdt", [("f32", "f32"), ("bf16", "f32"), ("f16", "f32"),
                                     ("bf16", "bf16"), ("f16", "f16"), ("f32", "f16")])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6])
def test_narrow_thread_mapped(cuda, oracle_mod, ragged, n, vdt, bdt):
    """A thread per row up to 5 columns: rows of 0 .. 12,000 nonzeros, all value
    and B types, scales; equal to the reference loop bit for bit."""
    from edge_loops_gb300 import api
    off, idx, vals = ragged
    dt = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
    g = torch.Generator(device=cuda)
    g.manual_seed(n)
    B = (torch.rand(20_000, n, device=cuda, generator=g) * 2 - 1).to(dt[bdt])
    A = api.CSR.from_arrays(off, idx, vals, 20_000, device=cuda)
    scale = None
    if vdt != "f32":
        A = A.quantized(dt[vdt])
        scale = A.row_scale.cpu().numpy()
    C = api.spmm(A, B, schedule="thread_mapped")
    assert api.workspace_errors() == 0
    exp = oracle_mod.spmm_f32(off, idx, A.values.float().cpu().numpy(), as_f32(B))
    if scale is not None:
        exp = exp * scale[:, None]  # powers of two: exact
    np.testing.assert_array_equal(C.cpu().numpy(), exp)
