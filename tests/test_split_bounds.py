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
    """split_nonzero of the bounded end, and of the end as the offsets have it."""
    n = d - w * x
    return tuple(min(n, e) if x < rows else n for e in (min(max(end, 0), nnz), end))


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
    outside = set()  # kinds whose coordinates leave [0, nnz] without the bounds
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


# ------------------------------------------------------------------- SpMM
BLOCK, MAX_NZ, ROW_ITEMS = 4096, 8192, 2  # spmm_impl.cuh
MAX_ROWS = BLOCK // ROW_ITEMS + 1
ENDS_WORDS, ROWM_WORDS = MAX_NZ // 32 + 4, MAX_ROWS // 32 + 4


def spmm_block(off, nnz, rs, re, ns, ne, inside, ordered, groups, u, long_row):
    """Walk::block: asserts what it reads and writes; the row it stops at."""
    rows = len(off) - 1
    assert 0 <= rs <= re <= rows and re - rs <= MAX_ROWS and 0 <= ns <= ne <= nnz
    assert ordered or ne - ns <= MAX_NZ
    nrows, length = re - rs, ne - ns
    assert (min(length, MAX_NZ) >> 5) + 2 <= ENDS_WORDS and (nrows >> 5) + 2 <= ROWM_WORDS
    if ordered:
        for i in range(nrows):
            s, e = int(off[rs + i]), int(off[rs + i + 1])
            if not 0 <= e - s <= long_row or not 0 <= e - ns <= MAX_NZ:
                nrows, ne = i, min(max(s, ns), ne)
                break
    ends, rowm, z_out = set(), [], False
    for i in range(nrows):
        s, e = int(off[rs + i]), int(off[rs + i + 1])
        z = not ordered and i == 0 and inside and e == ns
        z_out |= z
        if s != e and not z and ns < e <= ne and e - ns <= MAX_NZ:
            assert 0 <= (e - ns - 1) >> 5 < ENDS_WORDS
            ends.add(e - ns - 1)
            rowm.append(i)
    if ordered:
        re = rs + nrows
        if nrows == 0:
            return re
        ne = min(ne, ns + MAX_NZ)
    length = ne - ns
    per = -(-length // (groups * u)) * u
    dense = len(rowm) == nrows
    pieces = []
    for g in range(groups):
        q = min(per * g, length)
        assert (q >> 5) < ENDS_WORDS
        before = sum(e < q for e in ends)
        k = before if dense else (rowm[before] if before < len(rowm) else nrows)
        pieces.append((min(k, nrows) if not dense else k, ns + q))
    for g, (k, y) in enumerate(pieces):
        if ordered:  # whole rows, from row k's start to the next piece's row's
            def start(j):
                return min(max(int(off[rs + j]), ns), ne) if j < nrows else ne
            y = start(k)
            ye = max(start(pieces[g + 1][0]) if g + 1 < groups else ne, y)
        else:
            ye = min(y + per, ne)
        assert 0 <= y <= ye <= nnz and ye - ns <= MAX_NZ  # indices, values, M.ends
        for e in sorted(e for e in ends if y - ns <= e < ye - ns):
            assert k < nrows, "a store past the block's rows"
            k = k + 1 if dense else next((r for r in rowm if r > k), nrows)
    return re


def spmm_range(off, nnz, items, ordered, groups, u, long_row):
    """Every warp range of spmm_kernel, in blocks."""
    rows = len(off) - 1
    total = ROW_ITEMS * rows + nnz
    n_blocks = -(-items // BLOCK)
    block_items = -(-items // n_blocks)
    for d0 in range(0, total, items):
        d1 = min(d0 + items, total)
        for d in range(d0, d1, block_items):
            db = min(d + block_items, d1)
            rs, start, end = split(off, rows, nnz, d, ROW_ITEMS)
            re, start1, end1 = split(off, rows, nnz, db, ROW_ITEMS)
            ns = nonzero(rs, end, d, ROW_ITEMS, rows, nnz)[0]
            ne = nonzero(re, end1, db, ROW_ITEMS, rows, nnz)[0]
            re = min(max(re, rs), rs + MAX_ROWS)
            if not ordered:
                ne = min(max(ne, ns), ns + MAX_NZ)
                spmm_block(off, nnz, rs, re, ns, ne, ns > start, False, groups, u, long_row)
                continue
            ns = min(max(start, 0), nnz)
            ne = min(max(start1, ns), nnz)
            while rs < re:
                rs = spmm_block(off, nnz, rs, re, ns, ne, False, True, groups, u, long_row)
                if rs >= re:
                    break
                b = min(max(int(off[rs]), ns), ne)
                ns = min(max(int(off[rs + 1]), b), ne)
                assert 0 <= b <= ns <= nnz  # the long row's nonzeros
                rs += 1


@pytest.mark.parametrize("ordered", [False, True])
@pytest.mark.parametrize("groups,u", [(8, 4), (4, 8), (1, 8)])
def test_spmm_blocks_stay_inside(ordered, groups, u):
    rng = np.random.default_rng(5)
    for kind in KINDS + ["none"]:
        for rows, items in ((300, 64), (6000, 512), (6000, 9000), (9000, 4096)):
            off, nnz = offsets(kind, rng, rows)
            spmm_range(off, nnz, items, ordered, groups, u, 256 if groups > 1 else BLOCK)


def test_spmm_rows_of_two_split_points_were_unbounded():
    """What the bound on a block's rows is for: split points of offsets that
    are not monotone lie far apart."""
    off, nnz = offsets("random", np.random.default_rng(6), 60_000)
    most = 0
    for d in range(0, 2 * 60_000 + nnz - 4096, 4096):
        rs = split(off, 60_000, nnz, d, 2)[0]
        most = max(most, split(off, 60_000, nnz, d + 4096, 2)[0] - rs)
    assert most > 32 * ROWM_WORDS


def test_spmm_takes_the_bounded_coordinate():
    with open(os.path.join(CSRC, "spmm_impl.cuh")) as f:
        text = f.read()
    assert text.count("split_nonzero(") == 2 and "sp.end" not in text
    assert "min(max(re, rs), rs + kMaxRows)" in text and "min(max(ne, ns), ns + kMaxNz)" in text
