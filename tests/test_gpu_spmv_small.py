"""merge_path on small matrices, by both of its kernels: a CTA per range (the
default up to 8192 merge items per SM) and the warp walk (nz_per_lane=8 asks
for it at any size), at the sizes where the first can go wrong: one row, one
nonzero, ranges of one unit (256 items), more rows than the offsets it keeps
(4096), rows that are multiplied again from their start (up to 1024 nonzeros
earlier) and rows that wait for earlier ranges, empty rows, the switch between
the two.  Held to the order-free FP32 bound against FP64, and repeatable bit
for bit."""
import numpy as np
import pytest
import torch

from conftest import order_free_bound, random_csr

pytestmark = pytest.mark.gpu


def case(name, rng):
    if name == "one":
        return random_csr(rng, 1, 1, 1, long_rows=[(0, 1)])
    if name == "one_row":
        return random_csr(rng, 1, 60_000, 1, long_rows=[(0, 50_000)])
    if name == "unit":
        return random_csr(rng, 85, 300, 2)
    if name == "rows_4096":
        return random_csr(rng, 4096, 900, 9)
    if name == "rows_4097":
        return random_csr(rng, 4097, 900, 9, empty_frac=0.2)
    if name == "many_rows":
        return random_csr(rng, 60_000, 700, 3, empty_frac=0.5)
    if name == "again":  # rows around the 1024 that are multiplied again
        return random_csr(rng, 300, 9000, 30, long_rows=[(7, 1023), (30, 1024), (31, 1025),
                                                         (90, 1500), (150, 2000), (299, 1200)])
    if name == "long":
        return random_csr(rng, 40, 150_000, 5, long_rows=[(0, 9000), (3, 120_000), (39, 30_000)])
    if name == "empty":
        return random_csr(rng, 3000, 50, 0)
    if name == "mid":
        return random_csr(rng, 20_000, 5000, 26)
    if name == "last_small":  # just under 4 x 2048 items per SM (152 SMs), weight 2
        return random_csr(rng, 20_000, 5000, 116)
    return random_csr(rng, 21_500, 5000, 118)  # just over: the warp walk


NAMES = ["one", "one_row", "unit", "rows_4096", "rows_4097", "many_rows", "again", "long",
         "empty", "mid", "last_small", "first_walk"]


@pytest.mark.parametrize("dtype", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("opts", [{}, {"nz_per_lane": 8}, {"row_weight": 1}],
                         ids=["default", "walk", "weight1"])
@pytest.mark.parametrize("name", NAMES)
def test_bound_and_repeatable(cuda, oracle_mod, name, opts, dtype):
    from edge_loops_gb300 import api
    off, idx, vals, x = case(name, np.random.default_rng(NAMES.index(name)))
    A = api.CSR.from_arrays(off, idx, vals, len(x), device=cuda)
    scale = None
    if dtype != "f32":
        A = A.quantized(torch.bfloat16 if dtype == "bf16" else torch.float16)
        scale = A.row_scale.cpu().numpy()
    xt = torch.as_tensor(x, device=cuda)
    got = []
    for _ in range(2):
        y = torch.full((A.rows,), float("nan"), device=cuda)
        api.spmv(A, xt, y, **opts)
        got.append(y.cpu().numpy())
        assert api.workspace_errors() == 0
    np.testing.assert_array_equal(got[0], got[1])
    y64, yabs = oracle_mod.spmv_f64(off, idx, A.values.float().cpu().numpy(), x, row_scale=scale)
    assert np.all(np.abs(got[0] - y64) <= order_free_bound(off, yabs, extra=3))


@pytest.mark.parametrize("opts", [{}, {"nz_per_lane": 8}], ids=["default", "walk"])
def test_defects_are_flagged(cuda, opts):
    """Columns outside [0, cols) add nothing; offsets that fall, leave [0, nnz]
    or miss nnz raise a flag; every read stays inside the arrays (indices are
    clamped or checked before use)."""
    from edge_loops_gb300 import api
    off, idx, vals, x = random_csr(np.random.default_rng(3), 6000, 800, 12)
    xt = torch.as_tensor(x, device=cuda)

    def flags(o, i):
        A = api.CSR.from_arrays(o, i, vals, 800, device=cuda)
        y = api.spmv(A, xt, **opts)
        torch.cuda.synchronize()
        return api.workspace_errors(), y

    bad = idx.copy()
    bad[[0, 777, len(idx) - 1]] = [-1, 800, 2 ** 31 - 1]
    f, y = flags(off, bad)
    assert f == 1
    v0 = vals.copy()
    v0[[0, 777, len(idx) - 1]] = 0
    ref = api.spmv(api.CSR.from_arrays(off, idx, v0, 800, device=cuda), xt, **opts)
    assert torch.equal(y, ref)
    short = off.copy()
    short[-1] -= 3
    assert flags(short, idx)[0] & 6
    swapped = off.copy()
    swapped[3000], swapped[3001] = off[3001] + 9000, off[3000]
    assert flags(swapped, idx)[0] != 0
