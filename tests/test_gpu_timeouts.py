"""A look-back whose partials never come: every kernel that waits for earlier
ranges ends with EL_FLAG_TIMEOUT after its wait limit, and the workspace is
usable afterwards (the warp walk, the small kernel, work_oriented, SpMM)."""
import ctypes as C

import numpy as np
import pytest
import torch

from conftest import random_csr

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def long_row(cuda):
    from edge_loops_gb300 import api
    off, idx, vals, x = random_csr(np.random.default_rng(8), rows=10, cols=100_000, max_len=5,
                                   long_rows=[(4, 90_000)])
    return api.CSR.from_arrays(off, idx, vals, 100_000, device=cuda), torch.as_tensor(x, device=cuda)


def opts(**kw):
    from edge_loops_gb300 import api
    o = api.make_opts(wait_limit_us=2000, **kw)
    o.test_hooks = 1  # ranges do not publish their partials
    return o


@pytest.mark.parametrize("schedule,kw", [(0, {}), (0, {"nz_per_lane": 8}), (0, {"nz_per_lane": 16}),
                                         (1, {"num_threads": 512}), (0, {"compensated": True})],
                         ids=["small", "walk8", "walk16", "work_oriented", "compensated"])
def test_spmv(cuda, long_row, schedule, kw):
    from edge_loops_gb300 import _lib, api
    A, x = long_row
    y, ws, a = torch.empty(A.rows, device=cuda), api.Workspace(), A.el()
    st = _lib.lib().el_spmv(ws.handle, C.byref(a), schedule, C.byref(opts(**kw)),
                            C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr()),
                            C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == 0 and ws.errors() & _lib.EL_FLAG_TIMEOUT
    name = ["merge_path", "work_oriented"][schedule]
    again = api.spmv(A, x, y, schedule=name, workspace=ws, **kw)
    assert ws.errors() == 0
    assert torch.equal(again, api.spmv(A, x, schedule=name, **kw))


@pytest.mark.parametrize("n", [8, 24, 128])
def test_spmm(cuda, long_row, n):
    from edge_loops_gb300 import _lib, api
    A, _ = long_row
    B, ws, a = torch.rand(A.cols, n, device=cuda), api.Workspace(), A.el()
    out = torch.empty(A.rows, n, device=cuda)
    st = _lib.lib().el_spmm(ws.handle, C.byref(a), 0, C.byref(opts()), C.c_void_p(B.data_ptr()), 0,
                            n, n, C.c_void_p(out.data_ptr()), n,
                            C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == 0 and ws.errors() & _lib.EL_FLAG_TIMEOUT
    again = api.spmm(A, B, out, workspace=ws)
    assert ws.errors() == 0
    assert torch.equal(again, api.spmm(A, B))
