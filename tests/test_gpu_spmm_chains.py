"""The length of the SpMM walk's chains of additions (csrc/spmm_impl.cuh, kFold):
at most 33 steps of U nonzeros, also where the other lane groups of the warp
have a row end in every step.

Long rows hold 1 and then 1499 entries of 2^-25.  A chain that holds the 1 loses
every 2^-25 that is added to it (less than half a unit in the last place of 1),
and no other chain loses any, so a row's error counts the length of its first
chain."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

LONG, PAIRS, COLS = 1500, 2480, 64
TINY = 2.0 ** -25


@pytest.mark.parametrize("n,steps", [(16, 4), (32, 8), (64, 8), (128, 8)],
                         ids=["groups-of-4", "groups-of-8", "groups-of-16", "groups-of-32"])
def test_chains_are_short_beside_rows_of_one_nonzero(cuda, n, steps):
    """`steps`: nonzeros of a step, U.  Beside the first chain, a row's sum is
    rounded where its later parts are added to a sum of 1 or more: once per
    chain put aside, per piece and per range, each at most half a unit in the
    last place of 1, i.e. 2 x TINY."""
    from edge_loops_gb300 import api
    lens = torch.ones(PAIRS, LONG + 1, dtype=torch.int64, device=cuda)
    lens[:, 0] = LONG
    lens = lens.flatten()
    off = torch.zeros(lens.numel() + 1, dtype=torch.int64, device=cuda)
    off[1:] = torch.cumsum(lens, 0)
    nnz = int(off[-1])
    vals = torch.full((nnz,), TINY, device=cuda)
    first = off[:-1][:: LONG + 1]
    vals[first] = 1.0
    idx = torch.zeros(nnz, dtype=torch.int32, device=cuda)
    A = api.CSR(off.to(torch.int32), idx, vals, lens.numel(), COLS)
    C = api.spmm(A, torch.ones(COLS, n, device=cuda), schedule="merge_path")
    assert api.workspace_errors() == 0
    got = C.double()
    exact = 1.0 + (LONG - 1) * TINY
    short = torch.ones(lens.numel(), dtype=torch.bool, device=cuda)
    short[:: LONG + 1] = False
    assert bool((got[short] == TINY).all())
    lost = ((got[~short] - exact).abs().max() / TINY).item()
    chains = -(-LONG // (32 * steps)) + 1
    pieces = 2 + LONG // 128
    assert lost <= 33 * steps + 2 * (chains + pieces), lost
