"""Split points of the merge ranges on malformed offsets (csrc/el_device.cuh,
warp_merge_search2_w and split_nonzero), checked on the CPU: the 33-way search
restated probe by probe (on offsets that fall, which split it finds depends on
its probes) and run over offsets that are negative, too large, falling,
reversed or random.  Every range's nonzeros lie inside [0, nnz), every split
row inside [0, rows], and every offset that is read exists."""
import os

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "edge_loops_gb300", "csrc")


def split(off, rows, nnz, d, w):
    """warp_merge_search2_w for one diagonal: (x, offsets[x], offsets[x + 1])."""
    def row_end(k):
        assert -1 <= k < rows
        return int(off[k + 1])

    lo = min((d - nnz) // w if d > nnz else 0, rows)
    hi = min(d // w, rows)
    while hi - lo > 32:
        p = [lo + (lane + 1) * (hi - lo) // 33 for lane in range(32)]
        c = sum(row_end(q) <= d - w * (q + 1) for q in p)
        plo, phi = p[max(c - 1, 0)], p[min(c, 31)]
        if c > 0:
            lo = plo + 1
        if c < 32:
            hi = phi
    x = lo + sum(q < hi and row_end(q) <= d - w * (q + 1) for q in range(lo, lo + 32))
    return x, row_end(x - 1), row_end(x) if x < rows else nnz


def nonzero(x, end, d, w, rows, nnz):
    """split_nonzero, and the coordinate before its bounds."""
    n = d - w * x
    raw = min(n, end) if x < rows else n
    return min(max(raw, 0), nnz), raw


def ranges(off, nnz, w, items):
    """(rs, ns, re, ne, offsets[rs], raw ns, raw ne) of every range."""
    rows = len(off) - 1
    total = w * rows + nnz
    for d0 in range(0, total, items):
        d1 = min(d0 + items, total)
        rs, start, end = split(off, rows, nnz, d0, w)
        re, _, end1 = split(off, rows, nnz, d1, w)
        ns, raw0 = nonzero(rs, end, d0, w, rows, nnz)
        ne, raw1 = nonzero(re, end1, d1, w, rows, nnz)
        yield rs, ns, re, ne, start, raw0, raw1


def offsets(kind, rng, rows, mean=4):
    """Malformed offsets of a matrix of `rows` rows, and its nnz."""
    off = np.concatenate([[0], np.cumsum(rng.integers(0, 2 * mean + 1, rows))]).astype(np.int64)
    nnz = int(off[-1])
    k = rng.integers(1, max(rows, 2))
    if kind == "negative":
        off[k] = -50
    elif kind == "first row":
        off[1] = -50
    elif kind == "int min":
        off[k] = -2 ** 31
    elif kind == "too large":
        off[k:k + 40] = nnz + rng.integers(1, 100)
    elif kind == "int max":
        off[k] = 2 ** 31 - 1
    elif kind == "falls":
        off[k] = off[max(k - 700, 0)]
    elif kind == "reversed":
        off = off[::-1].copy()
    elif kind == "halves":
        off = np.concatenate([off[rows // 2:], off[:rows // 2]])
    elif kind == "random":
        off = rng.integers(0, nnz + 1, rows + 1)
    elif kind == "wild":
        off = rng.integers(-2 ** 31, 2 ** 31, rows + 1)
    elif kind == "all negative":
        off[1:] = -rng.integers(1, 2000, rows)
    elif kind == "short":
        off[-1] -= 3
    return off, nnz


KINDS = ["negative", "first row", "int min", "too large", "int max", "falls", "reversed", "halves",
         "random", "wild", "all negative", "short"]


def test_every_range_stays_inside():
    rng = np.random.default_rng(3)
    outside = set()  # kinds whose coordinates leave [0, nnz] before the bounds
    for kind in KINDS:
        for rows in (7, 300, 6000):
            for trial in range(12 if rows < 6000 else 3):
                off, nnz = offsets(kind, rng, rows)
                for w in (1, 2, 5):
                    for rs, ns, re, ne, start, raw0, raw1 in ranges(off, nnz, w, 256):
                        assert 0 <= rs <= rows and 0 <= re <= rows
                        assert 0 <= ns <= nnz and 0 <= ne <= nnz
                        if min(raw0, raw1) < 0 or max(raw0, raw1) > nnz:
                            outside.add(kind)
                        # the small kernel multiplies a row again from its
                        # start when that lies at most 1024 before the range
                        if ns > start and rs < re and start >= 0 and ns - start <= 1024:
                            assert 0 <= start <= nnz
    assert {"negative", "first row", "too large", "wild", "all negative"} <= outside


def test_well_formed_offsets_are_not_changed():
    rng = np.random.default_rng(4)
    for rows in (1, 33, 2000):
        off, nnz = offsets("none", rng, rows)
        for w in (1, 2, 16):
            last = (0, 0)
            for rs, ns, re, ne, start, raw0, raw1 in ranges(off, nnz, w, 512):
                assert (ns, ne) == (raw0, raw1) and (rs, ns) == last
                last = (re, ne)
            assert last == (rows, nnz)


@pytest.mark.parametrize("source", ["spmv_merge_path_nz.cuh", "spmv_merge_path_small.cuh"])
def test_kernels_take_the_bounded_coordinate(source):
    """No kernel forms the nonzero coordinate itself."""
    with open(os.path.join(CSRC, source)) as f:
        text = f.read()
    assert text.count("split_nonzero(") == 2
    assert "sp.end" not in text and "sa.end" not in text and "sb.end" not in text
