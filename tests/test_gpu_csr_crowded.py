"""el_csr_from_coo where a window overfills (a long row whose columns crowd
together): the pass that moves the entries stops at the first full window, and
the radix sort takes over without a second check of the entries.  The crowd
comes first, last or scattered in the COO, in small and large windows; one place
more or less than a window's room."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["first", "last", "scattered"])
@pytest.mark.parametrize("n,hub", [(60_000, 30_000), (60_000, 4096), (60_000, 4097),
                                   (2_200_000, 400_000), (2_200_000, 12_288), (2_200_000, 12_289)])
def test_crowded_row(cuda, n, hub, order):
    from edge_loops_gb300 import api
    rows, cols, g = 5000, 1 << 20, torch.Generator(device=cuda)
    g.manual_seed(n + hub)
    ri = torch.randint(0, rows, (n,), generator=g, device=cuda)
    ci = torch.randint(0, cols, (n,), generator=g, device=cuda)
    at = slice(0, hub) if order == "first" else slice(n - hub, n)
    ri[at] = rows // 3
    ci[at] = torch.randint(0, 300, (hub,), generator=g, device=cuda) + cols // 2
    if order == "scattered":
        p = torch.randperm(n, generator=g, device=cuda)
        ri, ci = ri[p], ci[p]
    vv = torch.rand(n, generator=g, device=cuda)
    A = api.csr_from_coo(rows, cols, ri.int(), ci.int(), vv)
    key, perm = torch.sort(ri * cols + ci, stable=True)
    off = torch.zeros(rows + 1, dtype=torch.int64, device=cuda)
    off[1:] = torch.cumsum(torch.bincount(ri, minlength=rows), 0)
    assert torch.equal(A.offsets.long(), off)
    assert torch.equal(A.indices.long(), key % cols)
    assert torch.equal(A.values, vv[perm])
    # an entry outside is still an error, whichever way is taken
    ci[n // 2] = cols
    with pytest.raises(Exception, match="MALFORMED"):
        api.csr_from_coo(rows, cols, ri.int(), ci.int(), vv)
