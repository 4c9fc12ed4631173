"""el_csr_from_coo over the shapes where its window sort can go wrong: sizes
around a window (2048, 8192 places) and around the switch between the two,
rows longer than a window's spare room, rows whose columns crowd together,
many equal entries, windows that overfill (the radix sort takes over), mostly
empty rows, entries already in order, more rows than the count's tables hold.  Equal to a stable sort by (row,
column), array for array."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def entries(kind, n, rows, cols, g, cuda):
    def rnd(hi, k=n):
        return torch.randint(0, hi, (k,), generator=g, device=cuda)
    ri, ci = rnd(rows), rnd(cols)
    if kind == "sorted":
        ri = torch.sort(ri)[0]
    elif kind == "one_row":
        ri = torch.full_like(ri, rows // 2)
    elif kind == "one_cell":
        ri, ci = torch.full_like(ri, rows - 1), torch.full_like(ci, cols - 1)
    elif kind == "three_columns":
        ci = rnd(min(3, cols)) * ((cols - 1) // 2)
    elif kind == "crowded":  # every row's entries within 40 columns
        ci = (ri * 13 + rnd(40)) % cols
    elif kind == "long_rows":  # half the entries in 20 rows
        ri[: n // 2] = rnd(20, n // 2) * (rows // 20)
    elif kind == "long_crowded":  # the same, in 16 columns
        ri[: n // 2] = rnd(20, n // 2) * (rows // 20)
        ci[: n // 2] = rnd(min(16, cols), n // 2)
    p = torch.randperm(n, generator=g, device=cuda) if kind != "sorted" else \
        torch.arange(n, device=cuda)
    return ri[p].int(), ci[p].int(), torch.rand(n, generator=g, device=cuda)


@pytest.mark.parametrize("kind,n,rows,cols", [
    ("random", 1, 1, 1), ("random", 7, 3, 5), ("random", 2047, 300, 300),
    ("random", 2048, 2048, 9), ("random", 2049, 50, 70), ("random", 4097, 9000, 9000),
    ("random", 40_000, 8192, 17), ("random", 40_000, 8193, 100_000),
    ("random", 2 ** 21, 70_000, 2 ** 31 - 1), ("random", 2 ** 21 + 1, 1 << 20, 60_000),
    ("random", 3_000_000, 2_000_000, 1000), ("random", 5000, 3_000_000, 100),
    ("sorted", 100_000, 5000, 5000), ("sorted", 2_500_000, 100_000, 5000),
    ("one_row", 60_000, 9, 1 << 20), ("one_row", 3_000_000, 20_000, 1 << 20),
    ("one_cell", 1500, 40, 40), ("one_cell", 9000, 40, 40), ("one_cell", 2_200_000, 9000, 40),
    ("three_columns", 300_000, 900, 7), ("crowded", 400_000, 4000, 1 << 20),
    ("crowded", 4_000_000, 10_000, 1 << 20), ("long_rows", 300_000, 50_000, 1 << 20),
    ("long_rows", 4_000_000, 50_000, 1 << 20), ("long_crowded", 300_000, 50_000, 1 << 20),
    ("long_crowded", 4_000_000, 50_000, 1 << 20)])
def test_equals_a_stable_sort(cuda, kind, n, rows, cols):
    from edge_loops_gb300 import api
    g = torch.Generator(device=cuda)
    g.manual_seed(n + rows)
    ri, ci, vv = entries(kind, n, rows, cols, g, cuda)
    keep = [t.clone() for t in (ri, ci, vv)]
    A = api.csr_from_coo(rows, cols, ri, ci, vv)
    key, order = torch.sort(ri.long() * cols + ci.long(), stable=True)
    off = torch.zeros(rows + 1, dtype=torch.int64, device=cuda)
    off[1:] = torch.cumsum(torch.bincount(ri.long(), minlength=rows), 0)
    assert torch.equal(A.offsets.long(), off)
    assert torch.equal(A.indices.long(), key % cols)
    assert torch.equal(A.values, vv[order])
    for t, k in zip((ri, ci, vv), keep):  # the COO is only read
        assert torch.equal(t, k)


@pytest.mark.parametrize("n,rows", [(3000, 100), (3000, 9000), (2_200_000, 9000)])
def test_entries_outside_leave_the_output_alone(cuda, n, rows):
    import ctypes as C
    from edge_loops_gb300 import _lib as L
    g = torch.Generator(device=cuda)
    g.manual_seed(1)
    ri, ci, vv = entries("random", n, rows, 500, g, cuda)
    for bad_r, bad_c in ((rows, 0), (-1, 0), (0, 500), (0, -2)):
        r, c = ri.clone(), ci.clone()
        r[n // 2], c[n // 2] = bad_r, bad_c
        coo = L.ElCoo()
        coo.rows, coo.cols, coo.nnz = rows, 500, n
        coo.row_indices, coo.col_indices, coo.values = r.data_ptr(), c.data_ptr(), vv.data_ptr()
        off = torch.full((rows + 1,), -7, dtype=torch.int32, device=cuda)
        idx = torch.full((n,), -7, dtype=torch.int32, device=cuda)
        val = torch.full((n,), -7.0, device=cuda)
        st = L.lib().el_csr_from_coo(None, C.byref(coo), C.c_void_p(off.data_ptr()),
                                     C.c_void_p(idx.data_ptr()), C.c_void_p(val.data_ptr()),
                                     C.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert st == L.EL_ERR_MALFORMED_CSR
        torch.cuda.synchronize()
        assert bool((off == -7).all()) and bool((idx == -7).all()) and bool((val == -7).all())


def test_two_streams_with_their_own_workspaces(cuda):
    """Calls on two streams share nothing: each uses its stream's workspace."""
    from edge_loops_gb300 import api
    g = torch.Generator(device=cuda)
    g.manual_seed(2)
    sets = [entries("random", 300_000, 20_000, 9000, g, cuda) for _ in range(2)]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in sets]
    got = []
    for s, (ri, ci, vv) in zip(streams, sets):
        with torch.cuda.stream(s):
            got.append(api.csr_from_coo(20_000, 9000, ri, ci, vv))
    torch.cuda.synchronize()
    for A, (ri, ci, vv) in zip(got, sets):
        key, order = torch.sort(ri.long() * 9000 + ci.long(), stable=True)
        assert torch.equal(A.indices.long(), key % 9000)
        assert torch.equal(A.values, vv[order])
    assert np.all(A.offsets.cpu().numpy()[1:] >= A.offsets.cpu().numpy()[:-1])
