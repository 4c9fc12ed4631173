"""group_mapped and work_oriented on the merge-path walk: rows around the
groups (32, 128, 256 rows, and the counts at which a warp takes more of a
group), rows and groups of no nonzeros, long rows, thread counts that cut the
merge anywhere.  Held to the order-free FP32 bound against FP64 and
repeatable bit for bit."""
import numpy as np
import pytest
import torch

from conftest import order_free_bound, random_csr

pytestmark = pytest.mark.gpu


def flat_csr(rng, rows, cols, max_len):
    """random_csr for many rows (columns may repeat within a row)."""
    lens = rng.integers(0, max_len + 1, size=rows)
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    idx = rng.integers(0, cols, size=off[-1]).astype(np.int32)
    return (off, idx, rng.uniform(-1, 1, size=off[-1]).astype(np.float32),
            rng.uniform(-1, 1, size=cols).astype(np.float32))


def case(name):
    rng = np.random.default_rng(len(name))
    if name.startswith("rows"):
        return random_csr(rng, int(name[4:]), 700, 20, empty_frac=0.2)
    if name == "long":
        return random_csr(rng, 400, 60_000, 6, long_rows=[(0, 5000), (33, 40_000), (399, 257)])
    if name == "empty":
        return random_csr(rng, 500, 10, 0)
    return flat_csr(rng, {"many": 400_000, "more": 800_000}[name], 3000, 7)


NAMES = ["rows1", "rows31", "rows32", "rows33", "rows128", "rows129", "rows256", "rows257",
         "rows5000", "long", "empty", "many", "more"]
CONFIGS = [("group_mapped", {}), ("group_mapped", {"group_rows": 32}),
           ("group_mapped", {"threads_per_block": 256}), ("group_mapped", {"compensated": True}),
           ("work_oriented", {}), ("work_oriented", {"num_threads": 128}),
           ("work_oriented", {"num_threads": 12_800}),
           ("work_oriented", {"num_threads": 640, "compensated": True})]


@pytest.mark.parametrize("sched,opts", CONFIGS, ids=lambda v: str(v))
@pytest.mark.parametrize("name", NAMES)
def test_bound_and_repeatable(cuda, oracle_mod, name, sched, opts):
    from edge_loops_gb300 import api
    off, idx, vals, x = case(name)
    A = api.CSR.from_arrays(off, idx, vals, len(x), device=cuda)
    xt = torch.as_tensor(x, device=cuda)
    y64, yabs = oracle_mod.spmv_f64(off, idx, vals, x)
    got = []
    for _ in range(2):
        y = torch.full((A.rows,), float("nan"), device=cuda)
        api.spmv(A, xt, y, schedule=sched, **opts)
        assert api.workspace_errors() == 0
        got.append(y.cpu().numpy())
    np.testing.assert_array_equal(got[0], got[1])
    assert np.all(np.abs(got[0] - y64) <= order_free_bound(off, yabs))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("sched", ["group_mapped", "work_oriented"])
@pytest.mark.parametrize("name", ["rows129", "rows5000", "long", "many"])
def test_16bit_values_with_scales(cuda, oracle_mod, name, sched, dtype):
    from edge_loops_gb300 import api
    off, idx, vals, x = case(name)
    A = api.CSR.from_arrays(off, idx, vals, len(x), device=cuda).quantized(dtype)
    y = api.spmv(A, torch.as_tensor(x, device=cuda), schedule=sched)
    assert api.workspace_errors() == 0
    y64, yabs = oracle_mod.spmv_f64(off, idx, A.values.float().cpu().numpy(), x,
                                    row_scale=A.row_scale.cpu().numpy())
    assert np.all(np.abs(y.cpu().numpy() - y64) <= order_free_bound(off, yabs, extra=3))


@pytest.mark.parametrize("num_threads", [8192 * 32, 8192 * 32 + 128, 8192 * 64, 8192 * 128])
def test_many_threads_under_capture(cuda, oracle_mod, num_threads):
    """A new workspace has the carry slots of every thread count up to
    8192 x 128: nothing is allocated under capture."""
    from edge_loops_gb300 import api
    off, idx, vals, x = case("more")
    A = api.CSR.from_arrays(off, idx, vals, len(x), device=cuda)
    xt = torch.as_tensor(x, device=cuda)
    y = torch.full((A.rows,), float("nan"), device=cuda)
    api.spmv(A, xt, y, schedule="work_oriented", workspace=api.Workspace())
    y.fill_(float("nan"))
    ws = api.Workspace()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        api.spmv(A, xt, y, schedule="work_oriented", workspace=ws, num_threads=num_threads)
    g.replay()
    torch.cuda.synchronize()
    assert ws.errors() == 0
    y64, yabs = oracle_mod.spmv_f64(off, idx, vals, x)
    assert np.all(np.abs(y.cpu().numpy() - y64) <= order_free_bound(off, yabs))


@pytest.mark.parametrize("sched,opts", [
    ("merge_path_flat", {"nz_per_lane": 8}), ("merge_path_flat", {"compensated": True}),
    ("work_oriented", {}), ("work_oriented", {"num_threads": 9600}), ("group_mapped", {})],
    ids=lambda v: str(v))
@pytest.mark.parametrize("n", [70_000, 1_300_000])
def test_row_of_many_ranges(cuda, oracle_mod, n, sched, opts):
    """One row in up to some thousand ranges, between short ones."""
    from edge_loops_gb300 import api
    rng = np.random.default_rng(n)
    lens = np.concatenate([np.full(50, 3), [n], np.full(50, 2)])
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    idx = rng.integers(0, 5000, size=off[-1]).astype(np.int32)
    vals = rng.uniform(-1, 1, size=off[-1]).astype(np.float32)
    x = rng.uniform(-1, 1, size=5000).astype(np.float32)
    A = api.CSR.from_arrays(off, idx, vals, 5000, device=cuda)
    y64, yabs = oracle_mod.spmv_f64(off, idx, vals, x)
    got = [api.spmv(A, torch.as_tensor(x, device=cuda), schedule=sched, **opts).cpu().numpy()
           for _ in range(2)]
    assert api.workspace_errors() == 0
    np.testing.assert_array_equal(got[0], got[1])
    assert np.all(np.abs(got[0] - y64) <= order_free_bound(off, yabs))


def test_num_threads_is_checked(cuda):
    from edge_loops_gb300 import _lib, api
    off, idx, vals, x = case("rows33")
    A = api.CSR.from_arrays(off, idx, vals, len(x), device=cuda)
    with pytest.raises(_lib.ElError) as e:
        api.spmv(A, torch.as_tensor(x, device=cuda), schedule="work_oriented", num_threads=100)
    assert e.value.status == _lib.EL_ERR_INVALID_ARGUMENT
