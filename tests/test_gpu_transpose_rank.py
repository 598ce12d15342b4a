"""Transpose where the second pass ranks by rows: chunks that span one round of
rows, several, and too many (ranked by ballots), chunks holding a repeated
column, buckets that start off a vector boundary, the most buckets."""

import numpy as np
import pytest

from cases import np_u16, np_u32, to_device_csr

pytestmark = pytest.mark.gpu


def _csr(rows, cols, per_row, seed, repeat=0, unsorted=False):
    rng = np.random.default_rng(seed)
    n = rng.poisson(per_row, rows)
    n[rng.integers(0, rows, rows // 3)] = 0
    row = np.repeat(np.arange(rows), n)
    col = rng.integers(0, cols, len(row))
    key = np.unique(row.astype(np.int64) * cols + col)  # each cell once, columns ascending
    row, col = (key // cols), (key % cols)
    if repeat:
        at = rng.choice(len(row), repeat, replace=False)
        row, col = np.insert(row, at, row[at]), np.insert(col, at, col[at])
    if unsorted:  # each row's columns in any order
        p = np.lexsort((rng.random(len(row)), row))
        row, col = row[p], col[p]
    ptr = np.zeros(rows + 1, np.uint32)
    np.cumsum(np.bincount(row, minlength=rows), out=ptr[1:])
    return ptr, col.astype(np.uint32), rng.integers(1, 60000, len(col)).astype(np.uint16)


@pytest.mark.parametrize("rows,cols,per_row,repeat,unsorted", [
    (700, 300, 60, 0, False),          # one round
    (6_000, 300, 9, 0, False),         # spans around the bitmap's 1,152 rows
    (6_000, 300, 9, 40, False),        # with repeated columns in most chunks
    (30_000, 300, 6.5, 0, True),       # two rounds, columns in any order; a sparse second bucket
    (40_000, 256, 3.3, 0, False),      # three rounds
    (40_000, 256, 3.3, 3, False),      # a repeated column in few chunks
    (30_000, 300, 3, 3, True),         # too sparse for the row ranking
    (60_000, 256, 0.5, 0, False),
    (60_000, 777, 2, 5, True),         # more than one bucket, sparse, repeated
    (1_153, 513, 30, 0, False),        # the span's edge, a bucket of one column
    (40, 262_144, 3_000, 0, False),    # the most buckets, chunks far from full
    (8_192, 1, 0.9, 0, False),         # one column
    (8_192, 3_000, 1.2, 4, True),      # tiles of thousands of rows: pointers searched
    (3, 100_000, 20_000, 0, False),    # rows of several tiles
])
def test_transpose_ranks(cuda, orc, rows, cols, per_row, repeat, unsorted):
    from cellshard_b200.device import transpose

    ptr, idx, val = _csr(rows, cols, per_row, rows + cols, repeat, unsorted)
    t = transpose(to_device_csr(rows, cols, ptr, idx, val))
    rptr, ridx, rval = orc.csr_transpose(rows, cols, ptr, idx, val)
    assert np.array_equal(np_u32(t.ptr), rptr)
    assert np.array_equal(np_u32(t.idx), ridx)
    assert np.array_equal(np_u16(t.val), rval)


@pytest.mark.parametrize("gap", [30_000, 100_000])
def test_gap_of_empty_rows_inside_a_tile(cuda, orc, gap):
    """Two rows of entries with thousands of empty rows between and after them."""
    from cellshard_b200.device import transpose

    cols = 600
    idx = np.concatenate([np.arange(0, cols, 2), np.arange(0, cols, 3)]).astype(np.uint32)
    ptr = np.zeros(gap + 8, np.uint32)
    ptr[3:gap], ptr[gap:] = 300, 500
    val = np.arange(1, 501, dtype=np.uint16)
    t = transpose(to_device_csr(gap + 7, cols, ptr, idx, val))
    rptr, ridx, rval = orc.csr_transpose(gap + 7, cols, ptr, idx, val)
    assert np.array_equal(np_u32(t.ptr), rptr) and np.array_equal(np_u32(t.idx), ridx)
    assert np.array_equal(np_u16(t.val), rval)


@pytest.mark.parametrize("n", [1_024 * 4_096, 1_024 * 4_096 + 1, 1_027 * 4_096 + 77])
def test_tiles_around_the_direct_offset_scan(cuda, n):
    """The most tiles whose offsets come from one kernel, and more."""
    from cellshard_b200.device import transpose

    rng = np.random.default_rng(n)
    rows, cols, per = 9_000, 1_500, n // 9_000
    count = np.full(rows, per)
    count[:n - per * rows] += 1
    ptr = np.concatenate([[0], np.cumsum(count)]).astype(np.uint32)
    first = rng.integers(0, cols, rows)
    within = np.arange(n) - np.repeat(ptr[:-1].astype(np.int64), count)
    idx = ((np.repeat(first, count) + within) % cols).astype(np.uint32)  # distinct in a row, in any order
    val = (np.arange(n) * 7 % 60_000).astype(np.uint16)
    t = transpose(to_device_csr(rows, cols, ptr, idx, val))
    order = np.argsort(idx, kind="stable")
    row = np.repeat(np.arange(rows, dtype=np.uint32), count)
    assert np.array_equal(np_u32(t.ptr), np.concatenate([[0], np.cumsum(np.bincount(idx, minlength=cols))]))
    assert np.array_equal(np_u32(t.idx), row[order]) and np.array_equal(np_u16(t.val), val[order])


@pytest.mark.parametrize("last,short", [
    ((1 << 24) - 2, 2),      # the last word of the range
    ((1 << 24) - 102, 2),    # the word before it
    ((1 << 24) - 620, 30),   # the first chunk start at which the word of all ones lies in the span
])
def test_most_rows(cuda, last, short):
    """2^24 - 1 rows; the last chunk, `short` entries below a whole one, ends in row `last`."""
    import torch

    from cellshard_b200.device import CSR, transpose

    rows, cols, chunk = (1 << 24) - 1, 256, 8_192
    # 3 entries in most rows, 16 in the last 600 that hold any; enough for the row ranking (3 a row)
    count = np.full(rows, 3, np.int64)
    count[last + 1:] = 0
    count[last - 599:last + 1] = 16
    need = max(0, 3 * rows - int(count.sum()))
    count[1:need + 2 * chunk:2] += 2
    over = (int(count.sum()) + short) % chunk  # one entry fewer in `over` early rows
    count[1:2 * over:2] -= 1
    n = int(count.sum())
    assert n % chunk == chunk - short and n >= 3 * rows
    ptr = np.concatenate([[0], np.cumsum(count)])
    row = torch.repeat_interleave(torch.arange(rows, device="cuda", dtype=torch.int32),
                                  torch.from_numpy(count).cuda())
    at = torch.arange(n, device="cuda") - torch.from_numpy(ptr[:-1]).cuda()[row.long()]
    col = ((row * 7 + at * 16 + 15) % cols).to(torch.int32)  # distinct in a row, in any order
    val = (torch.arange(n, device="cuda") % 30_011).to(torch.int16)
    t = transpose(CSR(rows, cols, torch.from_numpy(ptr.astype(np.uint32).view(np.int32)).cuda(), col,
                      val.view(torch.float16)))
    _, order = torch.sort(col.to(torch.uint8), stable=True)
    assert np.array_equal(np_u32(t.ptr), np.concatenate([[0], np.cumsum(np.bincount(col.cpu(), minlength=cols))]))
    assert torch.equal(t.idx, row[order]) and torch.equal(t.val.view(torch.int16), val[order])


@pytest.mark.parametrize("cols,n,skew", [
    (262_144, 300_000, 0.0),      # 1,024 buckets of a chunk each
    (262_144, 2_080_700, 0.9),    # the longest bucket that a thread per digit walks, nearly all entries in it
    (262_144, 2_089_000, 0.9),    # one more: in slices
    (262_144, 9_000_000, 0.5),
    (120_000, 900_000, 0.3),      # fewer chunks than one scan takes, either way
    (120_000, 980_000, 0.3),
    (16_000, 5_000_000, 0.0),     # few buckets
])
def test_offsets_of_many_buckets(cuda, cols, n, skew):
    """Second-pass offsets over many buckets, one of them holding up to nearly all entries."""
    import torch

    from cellshard_b200.device import CSR, transpose

    g = torch.Generator(device="cuda").manual_seed(n)
    rows = 4_000
    row = torch.sort(torch.randint(0, rows, (n,), generator=g, device="cuda")).values
    col = torch.randint(0, cols, (n,), generator=g, device="cuda")
    hot = torch.rand(n, generator=g, device="cuda") < skew
    col = torch.where(hot, col % 256 + 256 * 3, col)  # rows repeat columns; input order decides
    val = (torch.arange(n, device="cuda") % 30_011).to(torch.int16)
    ptr = torch.zeros(rows + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(torch.bincount(row, minlength=rows), 0, out=ptr[1:])
    t = transpose(CSR(rows, cols, ptr.to(torch.int32), col.to(torch.int32), val.view(torch.float16)))
    order = torch.sort(col, stable=True).indices
    assert torch.equal(t.ptr[1:].long(), torch.cumsum(torch.bincount(col, minlength=cols), 0))
    assert torch.equal(t.idx.long(), row[order]) and torch.equal(t.val.view(torch.int16), val[order])


@pytest.mark.parametrize("cols,sections", [
    (256, [(9_000, 9)]),                                       # a round a chunk, or two
    (256, [(20_000, 12), (20_000, 3.4), (9_000, 2.4)]),        # two and three rounds
    (256, [(30_000, 12), (25_000, 2.0), (2_000, 20)]),         # four, the most
    (256, [(30_000, 12), (25_000, 1.9), (25_000, 1.75)]),      # around the edge to five, ranked by ballots
    (256, [(30_000, 12), (4_600, 0), (9_000, 2.2), (70_000, 0.01), (40_000, 12)]),  # gaps of empty rows
    (300, [(30_000, 14), (15_000, 4.0)]),                      # a second bucket of 44 columns
    (1_000, [(12_000, 60), (12_000, 9)]),
    (262_144, [(40, 4_400)]),                                  # the most buckets
])
@pytest.mark.parametrize("repeat,unsorted", [(0, False), (0, True), (5, True), (2_000, False)])
def test_row_ranking_rounds(cuda, orc, cols, sections, repeat, unsorted):
    """Matrices that take the row ranking (three entries per row and 256 columns), with chunks of one
    to five rounds of 1,152 rows."""
    from cellshard_b200.device import transpose

    rows = sum(r for r, _ in sections)
    rng = np.random.default_rng(rows + cols + repeat)
    n = np.concatenate([rng.poisson(per, r) for r, per in sections])
    row = np.repeat(np.arange(rows), n)
    key = np.unique(row.astype(np.int64) * cols + rng.integers(0, cols, len(row)))
    row, col = key // cols, key % cols
    if repeat:
        at = rng.choice(len(row), repeat, replace=False)
        row, col = np.insert(row, at, row[at]), np.insert(col, at, col[at])
    if unsorted:
        p = np.lexsort((rng.random(len(row)), row))
        row, col = row[p], col[p]
    assert len(row) >= 3 * rows * -(-cols // 256)
    ptr = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=rows))]).astype(np.uint32)
    idx, val = col.astype(np.uint32), rng.integers(1, 60_000, len(col)).astype(np.uint16)
    t = transpose(to_device_csr(rows, cols, ptr, idx, val))
    rptr, ridx, rval = orc.csr_transpose(rows, cols, ptr, idx, val)
    assert np.array_equal(np_u32(t.ptr), rptr)
    assert np.array_equal(np_u32(t.idx), ridx)
    assert np.array_equal(np_u16(t.val), rval)
