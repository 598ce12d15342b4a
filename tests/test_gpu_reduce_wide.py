"""mask_groups reduce of CSR and Sliced-ELL rows with 15 to 32 groups (the
kernel that compacts the entries taking part in a group): the group counts at
its edges, rows that start and end anywhere in a vector, rows with more staged
entries than a step drains, tables at and past the shared-memory limit."""

import numpy as np
import pytest

from cases import np_u16, np_u32, to_device_csr

pytestmark = pytest.mark.gpu


def _inputs(rows, cols, longest, seed, in_groups, groups):
    rng = np.random.default_rng(seed)
    n = np.minimum(rng.integers(0, longest + 1, rows), cols)
    n[: min(rows, 12)] = np.minimum(np.arange(min(rows, 12)), cols)  # every short length once
    ptr = np.concatenate([[0], np.cumsum(n)]).astype(np.uint32)
    idx = np.concatenate([np.sort(rng.choice(cols, k, replace=False)) for k in n]).astype(np.uint32)
    val = rng.integers(0, 40, len(idx)).astype(np.float16)  # whole numbers, some zeros: sums are exact
    masks = rng.integers(0, 2 ** 32, cols, dtype=np.uint64).astype(np.uint32)
    masks[rng.random(cols) >= in_groups] = 0
    masks[rng.random(cols) < 0.02] = np.uint32(1 << (groups - 1))
    return ptr, idx, val.view(np.uint16), masks


@pytest.mark.parametrize("rows,cols,longest,groups,in_groups,masked", [
    (300, 900, 300, 15, 0.5, True),
    (300, 900, 300, 16, 0.5, True),
    (257, 900, 600, 17, 1.0, True),
    (257, 900, 600, 24, 0.0, False),
    (200, 5_000, 4_000, 31, 0.9, True),
    (200, 5_000, 4_000, 32, 0.9, True),
    (64, 5_000, 40, 32, 0.3, False),
    (40, 48_000, 900, 24, 0.5, True),   # a 192 KB table
    (40, 60_000, 900, 24, 0.5, True),   # past the shared memory: global tables
    (1, 3, 3, 20, 1.0, True),
])
@pytest.mark.parametrize("height", [0, 32, 5])
def test_many_groups(cuda, orc, rows, cols, longest, groups, in_groups, masked, height):
    import torch

    from cellshard_b200 import runtime
    from cellshard_b200.device import sliced_ell_from_csr

    ptr, idx, val, masks = _inputs(rows, cols, longest, rows + cols + groups, in_groups, groups)
    rng = np.random.default_rng(groups)
    rk = (rng.random(rows) < 0.8).astype(np.uint8) if masked else None
    fk = (rng.random(cols) < 0.7).astype(np.uint8) if masked else None
    filt = (20.0, 3, 0.6, groups - 1)

    def dev(a):
        return None if a is None else torch.from_numpy(a.copy()).cuda()

    src = to_device_csr(rows, cols, ptr, idx, val)
    if height:
        src = sliced_ell_from_csr(src, height)
        want = orc.group_reduce_sell(rows, cols, src.slice_rows, np_u32(src.slice_row_offsets),
                                     np_u32(src.slice_widths), np_u32(src.slice_slot_offsets), np_u32(src.col_idx),
                                     np_u16(src.val), masks, groups, rk, fk, filt)
    else:
        want = orc.group_reduce_csr(rows, cols, ptr, idx, val, masks, groups, rk, fk, filt)
    got = runtime.compute_sparse_group_reduce(src, dev(masks.view(np.int32)), groups, dev(rk), dev(fk),
                                              runtime.FilterParams(*filt))
    got = {k: v.cpu().numpy() for k, v in got.items()}
    for k in ("row_totals", "max_values", "row_keep", "group_counts", "group_percentages"):
        assert np.array_equal(got[k].reshape(-1), np.asarray(want[k]).reshape(-1)), k
    assert np.array_equal(got["detected_features"].view(np.uint32), want["detected_features"])


def _rows_csr(rows, cols, mean, seed):
    """mean +- half entries a row, columns ascending, one of each of `n` equal parts of the columns."""
    rng = np.random.default_rng(seed)
    n = np.minimum(rng.integers(mean // 2, mean + mean // 2 + 1, rows), cols)
    n[:12] = np.arange(12)
    ptr = np.concatenate([[0], np.cumsum(n)])
    row = np.repeat(np.arange(rows), n)
    j, k = np.arange(ptr[-1]) - ptr[row], n[row]
    lo, hi = j * cols // k, (j + 1) * cols // k
    return ptr.astype(np.uint32), (lo + rng.integers(0, 1 << 30, len(j)) % (hi - lo)).astype(np.uint32)


@pytest.mark.parametrize("rows,cols,mean,groups", [
    (20_000, 900, 45, 16),
    (10_000, 900, 30, 17),
    (10_000, 900, 30, 31),
    (12_000, 900, 40, 32),
    (1_500, 5_000, 1_200, 24),     # many sets of 16 a row
    (22_000, 40_703, 80, 17),      # around the widest table that fits
    (22_000, 40_704, 80, 24),
    (22_000, 40_705, 80, 31),      # past it: global tables
    (28_000, 39_469, 80, 32),      # with the bitmap behind it
    (28_000, 39_470, 80, 32),
    (28_000, 39_471, 80, 32),      # past it
])
@pytest.mark.parametrize("height", [0, 32])
def test_wide_route(cuda, orc, rows, cols, mean, groups, height):
    """Matrices large enough for the table (the rule of wide_pays, restated); the first rows alone
    are too few for it and give the same by the general kernel."""
    import torch

    from cellshard_b200 import runtime
    from cellshard_b200.device import sliced_ell_from_csr

    ptr, idx = _rows_csr(rows, cols, mean, rows + cols + groups)
    rng = np.random.default_rng(groups)
    val = rng.integers(0, 40, len(idx)).astype(np.float16).view(np.uint16)  # whole numbers: sums are exact
    masks = rng.integers(0, 2 ** 32, cols, dtype=np.uint64).astype(np.uint32)
    masks[rng.random(cols) < 0.4] = 0
    rk, fk = (rng.random(rows) < 0.8).astype(np.uint8), (rng.random(cols) < 0.7).astype(np.uint8)
    filt = (20.0, 3, 0.6, groups - 1)

    def pays(r, n):
        return 84 * r + n >= {16: 2.5, 32: 1.3}.get(groups, 1.0) * (0.9e6 + 60 * cols)

    def run(r):
        n = int(ptr[r])
        src = to_device_csr(r, cols, ptr[:r + 1], idx[:n], val[:n])
        if height:
            src = sliced_ell_from_csr(src, height)
        got = runtime.compute_sparse_group_reduce(src, torch.from_numpy(masks.view(np.int32)).cuda(), groups,
                                                  torch.from_numpy(rk[:r].copy()).cuda(), torch.from_numpy(fk).cuda(),
                                                  runtime.FilterParams(*filt))
        return {k: v.cpu().numpy().reshape(r, -1) for k, v in got.items()}

    few = 160
    assert pays(rows, int(ptr[rows])) and not pays(few, int(ptr[few]))
    got = run(rows)
    want = orc.group_reduce_csr(rows, cols, ptr, idx, val, masks, groups, rk, fk, filt)
    for k in ("row_totals", "max_values", "row_keep", "group_counts", "group_percentages"):
        assert np.array_equal(got[k].reshape(-1), np.asarray(want[k]).reshape(-1)), k
    assert np.array_equal(got["detected_features"].reshape(-1).view(np.uint32), want["detected_features"])
    for k, v in run(few).items():
        assert np.array_equal(v, got[k][:few]), k
