"""COO entries out of row order (put in row order by two counting-sort passes)
and CSR rows out of column order, to Blocked-ELL, against the restatement: the
edges of the 8,192-entry tiles, the low-digit widths, rows longer than a tile,
repeated cells near and far apart, and more rows than the passes take."""

import numpy as np
import pytest

from cases import np_u16, np_u32, to_device_csr

pytestmark = pytest.mark.gpu


def _entries(rows, cols, n, seed, hot=0, repeat=0):
    rng = np.random.default_rng(seed)
    row = rng.integers(0, rows, n).astype(np.uint32)
    col = rng.integers(0, cols, n).astype(np.uint32)
    if hot:  # one row holds most entries
        row[rng.random(n) < 0.8] = hot
    # distinct cells, then `repeat` copies of earlier cells at random later places
    _, first = np.unique(row.astype(np.int64) * cols + col, return_index=True)
    keep = rng.permutation(first)
    row, col = row[keep], col[keep]
    if repeat:
        k = rng.integers(0, len(row), repeat)
        at = np.sort(rng.integers(0, len(row) + 1, repeat))
        row, col = np.insert(row, at, row[k]), np.insert(col, at, col[k])
    val = rng.integers(1, 2000, len(row)).astype(np.float16)
    val[rng.random(len(row)) < 0.02] = 0
    return row, col, val.view(np.uint16)


@pytest.mark.parametrize("rows,cols,n,block,hot,repeat,remap", [
    (2, 9, 12, 8, 0, 0, False),
    (700, 900, 8_192, 16, 0, 0, False),          # one whole tile (before repeats fall out)
    (700, 900, 20_001, 16, 0, 300, True),        # repeats within a tile and across tiles
    (513, 40_000, 60_000, 16, 300, 20, False),   # a row of several tiles
    (262_144, 24, 30_000, 8, 0, 0, False),       # the most rows of an 8-bit low digit
    (262_145, 24, 30_000, 8, 0, 50, False),      # 9 bits
    (600_000, 24, 30_000, 8, 0, 0, True),        # 10 bits
    (1_300_000, 16, 30_000, 8, 0, 10, False),    # 11 bits
    (2_097_153, 8, 20_000, 8, 0, 10, False),     # past the partition: the sorts
])
def test_shuffled_coo(cuda, orc, rows, cols, n, block, hot, repeat, remap):
    import torch

    from cellshard_b200.device import blocked_ell_from_coo

    row, col, val = _entries(rows, cols, n, rows + n, hot, repeat)
    fmap = np.random.default_rng(1).permutation(cols).astype(np.uint32) if remap else None

    def dev(a, t):
        return torch.from_numpy(np.ascontiguousarray(a).view(t).copy()).cuda()

    out, counts, status, total = blocked_ell_from_coo(
        rows, cols, dev(row, np.int32), dev(col, np.int32), dev(val, np.float16), block, cols,
        dev(fmap, np.int32) if remap else None)
    ref = orc.blocked_ell_from_coo(rows, cols, row, col, val, block, fmap)
    assert status == 0 and out.ell_cols == ref["ell_cols"] and total == ref["total_blocks"]
    assert np.array_equal(np_u32(out.bci), ref["bci"])
    assert np.array_equal(np_u16(out.val), ref["val"])
    assert counts == [ref["nnz_host"], ref["nnz_gpu"]]


@pytest.mark.parametrize("cols,block,repeat", [
    (500, 8, False), (500, 8, True), (1_100, 24, True), (2_100, 16, False), (4_096, 16, True),  # a warp per row
    (4_104, 8, True), (9_000, 16, False), (9_000, 16, True), (16_384, 32, True),               # a CTA per row
    (32_768, 16, True), (32_768, 2, False),                                                    # one row buffer
    (333, 3, True), (40_000, 16, True),                                                        # no bulk stores
])
def test_csr_rows_in_any_column_order(cuda, orc, cols, block, repeat):
    from cellshard_b200.device import blocked_ell_from_csr

    rng = np.random.default_rng(cols + block)
    rows = 37
    parts = []
    for r in range(rows):
        # full row blocks of every kind: some rows past the 2,048 entries that registers hold
        c = rng.permutation(cols)[:int(rng.integers(0, min(cols, 5_000)))]
        if r % 3 == 0:
            c = np.sort(c)
        if repeat and r % 4 == 1 and len(c) > 1:
            c = np.append(c, c[rng.integers(0, len(c), 3)])
        parts.append(c)
    ptr = np.concatenate([[0], np.cumsum([len(c) for c in parts])]).astype(np.uint32)
    idx = np.concatenate(parts).astype(np.uint32)
    val = rng.integers(0, 2000, len(idx)).astype(np.float16).view(np.uint16)
    out = blocked_ell_from_csr(to_device_csr(rows, cols, ptr, idx, val), block)
    ref = orc.blocked_ell_from_csr(rows, cols, ptr, idx, val, block)
    assert out.ell_cols == ref["ell_cols"] and out.nnz == ref["nnz"]
    assert np.array_equal(np_u32(out.bci), ref["bci"]) and np.array_equal(np_u16(out.val), ref["val"])


@pytest.mark.parametrize("rows,cols,longest", [(1, 900, 900), (70, 6_100, 700), (5_000, 1_000, 40), (9_001, 300, 290)])
@pytest.mark.parametrize("block", [8, 24])
def test_short_rows_in_runs(cuda, orc, rows, cols, longest, block):
    """A warp per row: runs of rows over row-block borders, rows past 256 entries."""
    from cellshard_b200.device import blocked_ell_from_csr

    rng = np.random.default_rng(rows + block)
    n = rng.integers(0, longest + 1, rows)
    n[rng.random(rows) < 0.1] = longest
    ptr = np.concatenate([[0], np.cumsum(n)]).astype(np.uint32)
    idx = np.concatenate([np.sort(rng.choice(cols, k, replace=False)) for k in n]).astype(np.uint32)
    val = rng.integers(0, 60_000, len(idx)).astype(np.uint16)
    out = blocked_ell_from_csr(to_device_csr(rows, cols, ptr, idx, val), block)
    ref = orc.blocked_ell_from_csr(rows, cols, ptr, idx, val, block)
    assert out.ell_cols == ref["ell_cols"] and out.nnz == ref["nnz"]
    assert np.array_equal(np_u32(out.bci), ref["bci"]) and np.array_equal(np_u16(out.val), ref["val"])


@pytest.mark.parametrize("rows,cols,n,block,repeat", [
    (300, 1_000, 60_000, 1, 0), (300, 1_000, 60_000, 1, 3),  # one row per row block: one warp
    (301, 1_003, 90_000, 3, 1),                              # no power of two
    (90, 2_049, 80_000, 32, 0), (90, 2_049, 80_000, 32, 2),  # rows of several 256-column rounds
    (40, 203_000, 30_000, 16, 2),                            # the widest rows of which bitmaps fit, and
    (40, 210_000, 30_000, 16, 0), (40, 210_000, 30_000, 16, 2),  # wider: in the entries' order at once
])
def test_shuffled_coo_repeats_in_the_shape_pass(cuda, orc, rows, cols, n, block, repeat):
    test_shuffled_coo(cuda, orc, rows, cols, n, block, 0, repeat, False)


@pytest.mark.parametrize("n,repeat", [(8_390_000, 0), (8_800_000, 2)])
def test_shuffled_coo_of_many_tiles(cuda, orc, n, repeat):
    """Around 1,024 tiles of 8,192 entries: offsets by one kernel or in slices."""
    test_shuffled_coo(cuda, orc, 700, 100_000, n, 16, 0, repeat, False)


def test_shuffled_coo_past_the_column_blocks_is_refused(cuda):
    """131,072 column blocks at most, in any order of the entries."""
    import torch

    from cellshard_b200 import _abi
    from cellshard_b200.device import blocked_ell_from_coo

    row, col, val = _entries(40, 140_000, 30_000, 5)
    for order in (np.arange(len(row)), np.argsort(row, kind="stable")):
        dev = [torch.from_numpy(a[order].view(t).copy()).cuda()
               for a, t in ((row, np.int32), (col, np.int32), (val, np.float16))]
        with pytest.raises(_abi.CellShardError, match="column-block limit"):
            blocked_ell_from_coo(40, 140_000, *dev, 1, 140_000)


@pytest.mark.parametrize("cols,block", [
    (1_100, 24), (9_000, 16),               # rows by a warp, by a CTA
    (333, 3), (1_201, 1), (40_000, 16),     # no bulk stores: odd row sizes, two segments
])
@pytest.mark.parametrize("equal", [False, True])
def test_rows_that_repeat_a_column(cuda, orc, cols, block, equal):
    """Repeated columns with other values, the same one, NaN and zeros among them, in any order: the
    last value stays, and a cell counts once."""
    from cellshard_b200.device import blocked_ell_from_csr

    rng = np.random.default_rng(cols + block)
    rows = 61
    parts, vals = [], []
    for r in range(rows):
        c = rng.permutation(cols)[:int(rng.integers(1, min(cols, 3_000)))]
        v = rng.integers(0, 3, len(c)).astype(np.float16)
        v[rng.random(len(c)) < 0.05] = np.nan
        if r % 3:
            k = rng.integers(0, len(c), 4)
            more = v[k] if equal else rng.integers(0, 5, 4).astype(np.float16)
            p = rng.permutation(len(c) + 4)
            c, v = np.append(c, c[k])[p], np.append(v, more)[p]
        if r % 5 == 0:  # next to each other
            o = np.argsort(c, kind="stable")
            c, v = c[o], v[o]
        parts.append(c)
        vals.append(v)
    ptr = np.concatenate([[0], np.cumsum([len(c) for c in parts])]).astype(np.uint32)
    idx, val = np.concatenate(parts).astype(np.uint32), np.concatenate(vals).view(np.uint16)
    out = blocked_ell_from_csr(to_device_csr(rows, cols, ptr, idx, val), block)
    ref = orc.blocked_ell_from_csr(rows, cols, ptr, idx, val, block)
    assert out.ell_cols == ref["ell_cols"] and out.nnz == ref["nnz"]
    assert np.array_equal(np_u32(out.bci), ref["bci"]) and np.array_equal(np_u16(out.val), ref["val"])
