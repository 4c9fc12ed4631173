"""The SpMM look-back (csrc/spmm_impl.cuh): lane l of a warp acquires the flag
of range base + l, then every lane reads the vectors of all 32 ranges.  A warp
vote gives no memory ordering, so a __syncwarp() has to stand between the
acquires and the reads (a data race shows in no run that happens to be fine,
hence the check of the source); and a row that crosses hundreds of ranges is
summed the same in every call."""
import os

import numpy as np
import pytest
import torch

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "edge_loops_gb300", "csrc")


def test_the_reads_are_ordered_after_the_acquires():
    with open(os.path.join(CSRC, "spmm_impl.cuh")) as f:
        text = f.read()
    acquire = text.index("ld_acquire_u32(f)")
    read = text.index("const float* const src = a.vec")
    assert "__syncwarp();" in text[acquire:read]


@pytest.mark.gpu
@pytest.mark.parametrize("n", [8, 32, 128])
def test_a_row_over_many_ranges_is_the_same_each_time(cuda, oracle_mod, n):
    from edge_loops_gb300 import api
    rng = np.random.default_rng(n)
    cols, lens = 4000, np.array([3] * 50 + [300_000] + [5] * 50 + [70_000] + [2] * 50)
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    idx = rng.integers(0, cols, off[-1]).astype(np.int32)
    vals = rng.uniform(-1, 1, off[-1]).astype(np.float32)
    A = api.CSR.from_arrays(off, idx, vals, cols, device=cuda)
    B = rng.uniform(-1, 1, (cols, n)).astype(np.float32)
    Bt, first = torch.as_tensor(B, device=cuda), None
    for _ in range(20):
        C = api.spmm(A, Bt, schedule="merge_path")
        first = C if first is None else first
        assert torch.equal(C, first)
    assert api.workspace_errors() == 0
    C64, Ca = oracle_mod.spmm_f64(off, idx, vals, B)
    k = (lens + 2)[:, None]
    assert np.all(np.abs(first.cpu().numpy() - C64) <= k * 2.0 ** -24 / (1 - k * 2.0 ** -24) * Ca)
