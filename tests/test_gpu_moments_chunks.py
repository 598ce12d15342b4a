"""Grouped moments where the default chunk size differs (64 rows on small
matrices up to 2,048): whole counts, so every sum is exact in 64 bits; the
allocation-free entry point accepts what its static scratch always held."""

import ctypes as C

import numpy as np
import pytest

from cases import random_csr, to_device_csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,density,block,groups", [
    (1, 40, 0.5, 8, 3),
    (2_047, 333, 0.05, 16, 1),
    (5_000, 2_100, 0.01, 32, 300),
    (20_000, 700, 0.02, 8, 2),
    (3_001, 9_000, 0.004, 16, 5),
])
def test_default_chunks(cuda, rows, cols, density, block, groups):
    import torch

    from cellshard_b200 import _abi, runtime
    from cellshard_b200.device import blocked_ell_from_csr, ptr as dptr, stream_handle

    p, idx, val = random_csr(rows, cols, density, rows, 0.1)
    bell = blocked_ell_from_csr(to_device_csr(rows, cols, p, idx, val), block)
    rng = np.random.default_rng(rows)
    keep, lab = rng.random(rows) < 0.8, rng.integers(0, groups, rows)
    rk = torch.from_numpy(keep.astype(np.uint8)).cuda()
    labels = torch.from_numpy(lab.astype(np.int32)).cuda()
    row = np.repeat(np.arange(rows), np.diff(p.astype(np.int64)))
    x = val.view(np.float16).astype(np.float64)
    ok = keep[row]
    want = [np.zeros((groups, cols)), np.zeros((groups, cols))]
    for w, v in zip(want, (x, x * x)):
        np.add.at(w, (lab[row][ok], idx[ok].astype(np.int64)), v[ok])
    got = runtime.compute_sparse_group_moments(bell, groups, rk, None, labels)
    for w, k in zip(want, ("sum", "sumsq")):
        assert np.array_equal(got[k].cpu().numpy().astype(np.float64), w), k  # below 2^24: exact in fp32
    assert np.array_equal(got["group_rows"].cpu().numpy(), np.bincount(lab[keep], minlength=groups))
    if bell.ell_cols == 0:
        return
    lib = _abi.load()
    out = {k: torch.empty(groups, cols, device="cuda") for k in ("sum", "sumsq")}
    o = _abi.GroupMomentsOut(dptr(out["sum"]), dptr(out["sumsq"]))
    prm, v = _abi.GroupMomentsParams(groups, 2, 1, 0), bell.view()
    n = C.c_size_t()
    old = _abi.GroupMomentsParams(groups, 2, 1, 2048)
    _abi.check(lib.cs_b200_group_moments_scratch_bytes(C.byref(v), C.byref(old), C.byref(n)), "scratch")
    done = lib.cs_b200_group_moments_blocked_ell_noalloc(C.byref(v), dptr(rk), None, dptr(labels), C.byref(prm),
                                                         C.byref(o), stream_handle())
    assert done == (1 if n.value <= 64 << 20 else 0)
    if done:
        for w, k in zip(want, ("sum", "sumsq")):
            assert np.array_equal(out[k].cpu().numpy().astype(np.float64), w), k


@pytest.mark.parametrize("rows,cols,groups,chunk", [(8_192, 2_000, 8, 0), (3_000, 700, 9, 0), (3_000, 700, 9, 96),
                                                    (3_000, 4_000, 250, 0)])
def test_noalloc_gives_the_same_bits(cuda, rows, cols, groups, chunk):
    """Values that are no whole numbers: the order of the sums shows in the 64-bit results."""
    import torch

    from cellshard_b200 import _abi
    from cellshard_b200.device import blocked_ell_from_csr, ptr as dptr, stream_handle

    p, idx, val = random_csr(rows, cols, 0.06, rows, 0.1, integer=False)
    bell = blocked_ell_from_csr(to_device_csr(rows, cols, p, idx, val), 16)
    lab = torch.from_numpy(np.random.default_rng(rows).integers(0, groups, rows).astype(np.int32)).cuda()
    lib = _abi.load()
    v, prm, n = bell.view(), _abi.GroupMomentsParams(groups, 2, 1, chunk), C.c_size_t()
    _abi.check(lib.cs_b200_group_moments_scratch_bytes(C.byref(v), C.byref(prm), C.byref(n)), "scratch")
    assert n.value <= 64 << 20
    scratch = torch.empty(n.value, dtype=torch.uint8, device="cuda")
    got = []
    for noalloc in (False, True):
        out = [torch.zeros(groups, cols, dtype=t, device="cuda") for t in 4 * [torch.float32] + 2 * [torch.float64]]
        o = _abi.GroupMomentsOut(*(dptr(t) for t in out))
        if noalloc:
            ok = lib.cs_b200_group_moments_blocked_ell_noalloc(C.byref(v), None, None, dptr(lab), C.byref(prm),
                                                               C.byref(o), stream_handle())
        else:
            ok = lib.cs_b200_group_moments_blocked_ell(C.byref(v), None, None, dptr(lab), C.byref(prm), C.byref(o),
                                                       dptr(scratch), n.value, stream_handle())
        _abi.check(ok, "group_moments")
        got.append(out)
    assert float(got[0][0].abs().sum()) > 0
    for a, b in zip(*got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("groups", [1, 3, 1_024, 1_025, 2_000])
@pytest.mark.parametrize("chunk", [0, 64])
@pytest.mark.parametrize("scheme", [0, 1, 2])
def test_groups_of_many_chunks(cuda, groups, chunk, scheme):
    """Most rows in the first and the last group, groups of none between them: chunks cut by a thread
    each, over the 1,024 groups of a pass too, and combined in batches.  Whole counts: exact sums."""
    import torch

    from cellshard_b200 import runtime
    from cellshard_b200.device import blocked_ell_from_csr

    rows, cols = 9_001, 300
    p, idx, val = random_csr(rows, cols, 0.03, groups, 0.1)
    bell = blocked_ell_from_csr(to_device_csr(rows, cols, p, idx, val), 8)
    rng = np.random.default_rng(groups)
    lab = rng.integers(0, groups, rows) // 2 * 2
    lab[rng.random(rows) < 0.4] = 0
    lab[rng.random(rows) < 0.4] = groups - 1
    row = np.repeat(np.arange(rows), np.diff(p.astype(np.int64)))
    x = val.view(np.float16).astype(np.float64)
    got = runtime.compute_sparse_group_moments(bell, groups, None, None,
                                               torch.from_numpy(lab.astype(np.int32)).cuda(), scheme=scheme,
                                               chunk_rows=chunk)
    for k, v in (("sum", x), ("sumsq", x * x)):
        want = np.zeros((groups, cols))
        np.add.at(want, (lab[row], idx.astype(np.int64)), v)
        assert np.array_equal(got[k].cpu().numpy().astype(np.float64), want), k
    assert np.array_equal(got["group_rows"].cpu().numpy(), np.bincount(lab, minlength=groups))
