"""Execution buckets of a Sliced-ELL partition where the split over distinct
widths could go wrong: few widths with many ties, one width, as many widths as
buckets, widths past the row count, live slots behind padding."""

import numpy as np
import pytest

from cases import np_u16, np_u32
from test_gpu_exec_bucket import _dev_sell, _flat

pytestmark = pytest.mark.gpu
INVALID = 0xFFFFFFFF


def _part(row_widths, h, cols, seed, gaps):
    """Sliced-ELL with the given live slots per row; with gaps, padding stands between them."""
    rng = np.random.default_rng(seed)
    rows = len(row_widths)
    offsets = np.minimum(np.arange(0, rows + h, h), rows)
    widths, col, val = [], [], []
    for a, b in zip(offsets, offsets[1:]):
        w = int(max(row_widths[a:b])) + (3 if gaps else 0)
        widths.append(w)
        for r in range(a, b):
            c = np.full(w, INVALID, np.uint32)
            v = np.zeros(w, np.uint16)
            n = int(row_widths[r])
            at = np.sort(rng.choice(w, n, replace=False)) if gaps else np.arange(n)
            c[at] = np.sort(rng.choice(cols, n, replace=False))
            v[at] = rng.integers(1, 60000, n)
            col.append(c)
            val.append(v)
    return offsets, np.array(widths), np.concatenate(col), np.concatenate(val)


@pytest.mark.parametrize("kind,rows,h,gaps", [
    ("ties", 500, 16, False),
    ("ties", 500, 16, True),
    ("one", 300, 32, False),      # fewer widths than buckets
    ("eight", 400, 8, False),     # exactly as many
    ("nine", 400, 8, True),
    ("spread", 2_000, 32, False),
    ("wide", 20, 4, True),        # widths past the row count: no histogram
])
def test_split_by_widths(cuda, orc, kind, rows, h, gaps):
    from cellshard_b200.device import bucketed_sliced_ell

    rng = np.random.default_rng(rows + h)
    w = {"ties": rng.choice([0, 1, 2, 3, 5, 8, 8, 8, 40, 41], rows), "one": np.full(rows, 7),
         "eight": rng.integers(1, 9, rows) * 5, "nine": rng.integers(0, 9, rows),
         "spread": np.minimum(rng.lognormal(3.5, 0.8, rows), 300).astype(int),
         "wide": rng.integers(30, 400, rows)}[kind]
    offsets, widths, col, val = _part(w, h, 1_000, rows, gaps)
    sell = _dev_sell(rows, 1_000, int(w.sum()), offsets, widths, col, val)
    for req in (1, 2, 3, 8, 12, 0):
        bp = bucketed_sliced_ell(sell, req)
        want = req if req else orc.sell_choose_bucket_count(rows, offsets, widths, col)[0]
        ref = orc.sell_bucketed(rows, offsets, widths, col, val, want)
        assert bp.plan["segment_count"] == ref["segment_count"] and bp.plan["bytes"] == ref["bytes"], req
        assert bp.segment_row_offsets == list(ref["seg_row"].astype(int)), req
        got_col, got_val = _flat(bp)
        assert np.array_equal(got_col, ref["seg_col"]) and np.array_equal(got_val, ref["seg_val"]), req
        assert np.array_equal(np_u32(bp.exec_to_canonical_rows), ref["e2c"])
        assert np.array_equal(np_u32(bp.canonical_to_exec_rows), ref["c2e"])
        assert [int(np_u32(s.slice_widths)[0]) for s in bp.segments] == [s.col_idx.numel() // s.rows if s.rows else 0
                                                                         for s in bp.segments]
        assert np_u16(bp.val).size >= bp.plan["value_entries"]


@pytest.mark.parametrize("requested", [3, 4, 512])
def test_more_buckets_than_widths_of_many_rows(cuda, requested):
    """A million rows of three widths: one segment per width, however many are asked
    for, without a programme over the rows (512 levels of it take seconds)."""
    import time

    import torch

    from cellshard_b200.device import SlicedELL, bucketed_sliced_ell

    rows, w = 1_000_000, 4
    live = torch.randint(0, 3, (rows,), generator=torch.Generator().manual_seed(1)) + 1  # 1..3 of the slice's 4 slots
    col = torch.where(torch.arange(w)[None, :] < live[:, None], torch.arange(w, dtype=torch.int32)[None, :],
                      torch.full((), -1, dtype=torch.int32)).reshape(-1).cuda()
    val = torch.ones(rows * w, dtype=torch.float16, device="cuda")
    one = [torch.tensor(x, dtype=torch.int32, device="cuda") for x in ([0, rows], [w], [0])]
    sell = SlicedELL(rows, 9, int(live.sum()), rows, *one, col, val)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    bp = bucketed_sliced_ell(sell, requested)
    torch.cuda.synchronize()
    assert time.perf_counter() - t0 < 0.5
    n = torch.bincount(live, minlength=4)[1:].tolist()
    assert bp.segment_row_offsets == [0, n[0], n[0] + n[1], rows]
    assert [s.col_idx.numel() for s in bp.segments] == [n[0], 2 * n[1], 3 * n[2]]
    order = torch.argsort(live, stable=True)
    assert np.array_equal(np_u32(bp.exec_to_canonical_rows), order.numpy())
    for k, s in enumerate(bp.segments):
        assert torch.equal(s.col_idx.view(-1, k + 1), torch.arange(k + 1, dtype=torch.int32, device="cuda").expand(n[k], -1))
