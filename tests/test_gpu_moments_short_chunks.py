"""Grouped moments of groups of few rows (16-byte partial stores, four columns a
thread in the combine): ragged column counts, segments of every width, mean and
variance against 64-bit arithmetic, and scratch without room for the padding."""

import ctypes as C

import numpy as np
import pytest

from cases import random_csr, to_device_csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,block,groups", [
    (900, 1, 8, 300), (900, 1_023, 8, 300), (900, 1_025, 24, 297), (700, 3_001, 4, 250), (700, 2_050, 2, 250),
    (640, 517, 3, 300), (40, 20_011, 32, 17), (20_000, 130, 16, 39), (21_000, 130, 16, 40),
])
def test_short_chunks(cuda, rows, cols, block, groups):
    import torch

    from cellshard_b200 import _abi
    from cellshard_b200.device import blocked_ell_from_csr, ptr as dptr, stream_handle

    p, idx, val = random_csr(rows, cols, 0.05 if cols > 100 else 0.5, rows + cols, 0.1)
    bell = blocked_ell_from_csr(to_device_csr(rows, cols, p, idx, val), block)
    rng = np.random.default_rng(cols)
    keep, lab = rng.random(rows) < 0.9, rng.integers(0, groups, rows)
    fkeep = rng.random(cols) < 0.7
    rk, fk = (torch.from_numpy(a.astype(np.uint8)).cuda() for a in (keep, fkeep))
    labels = torch.from_numpy(lab.astype(np.int32)).cuda()
    row = np.repeat(np.arange(rows), np.diff(p.astype(np.int64)))
    x = val.view(np.float16).astype(np.float64)
    ok = keep[row] & fkeep[idx]
    s, q = np.zeros((groups, cols)), np.zeros((groups, cols))
    for w, v in ((s, x), (q, x * x)):
        np.add.at(w, (lab[row][ok], idx[ok].astype(np.int64)), v[ok])
    n = np.bincount(lab[keep], minlength=groups).astype(np.float64)[:, None]
    # whole counts: sums are exact, so mean and variance are one rounding sequence of doubles
    with np.errstate(divide="ignore", invalid="ignore"):
        mean = np.where(n > 0, s / n, 0.0)
        var = np.where(n > 1, np.maximum(q - s * mean, 0.0) / (n - 1.0), 0.0)
    lib = _abi.load()
    v, prm = bell.view(), _abi.GroupMomentsParams(groups, 2, 1, 0)
    need = C.c_size_t()
    _abi.check(lib.cs_b200_group_moments_scratch_bytes(C.byref(v), C.byref(prm), C.byref(need)), "scratch")
    for room in (need.value, need.value - (4 if cols % 8 else 0)):  # the second without room for the padding
        scratch = torch.full((room,), 0xff, dtype=torch.uint8, device="cuda")
        out = {k: torch.full((groups, cols), -1.0, dtype=t, device="cuda")
               for k, t in (("sum", torch.float32), ("sumsq", torch.float32), ("mean", torch.float32),
                            ("var", torch.float32), ("mean64", torch.float64), ("var64", torch.float64))}
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        o = _abi.GroupMomentsOut(dptr(out["sum"]), dptr(out["sumsq"]), dptr(out["mean"]), dptr(out["var"]))
        o.mean64, o.var64, o.status = dptr(out["mean64"]), dptr(out["var64"]), dptr(status)
        _abi.check(lib.cs_b200_group_moments_blocked_ell(C.byref(v), dptr(rk), dptr(fk), dptr(labels), C.byref(prm),
                                                         C.byref(o), dptr(scratch), room, stream_handle()), "moments")
        got = {k: t.cpu().numpy() for k, t in out.items()}
        assert np.array_equal(got["sum"], s.astype(np.float32)) and np.array_equal(got["sumsq"], q.astype(np.float32))
        assert np.array_equal(got["mean64"], mean)
        # q - s * mean may be contracted: one rounding of s * mean apart
        tol = 2.0 ** -52 * np.abs(s * mean) / np.maximum(n - 1.0, 1.0) + 2.0 ** -51 * var
        assert np.all(np.abs(got["var64"] - var) <= tol)
        assert np.array_equal(got["mean"], mean.astype(np.float32))


@pytest.mark.parametrize("rows,cols", [(8_000, 900), (8_000, 901), (3_000, 2_003)])
def test_scratch_sized_for_longer_chunks(cuda, rows, cols):
    """Scratch for chunks of 512 or 2,048 rows, padded or not, does where the
    default is 64: the sums are those of the full scratch."""
    import torch

    from cellshard_b200 import _abi
    from cellshard_b200.device import blocked_ell_from_csr, ptr as dptr, stream_handle

    lib = _abi.load()
    p, idx, val = random_csr(rows, cols, 0.03, rows + cols, 0.1)
    bell = blocked_ell_from_csr(to_device_csr(rows, cols, p, idx, val), 16)
    labels = torch.arange(rows, dtype=torch.int32, device="cuda") % 3
    v = bell.view()
    parts = (_abi.BlockedEllView * 1)(v)

    def need(chunk, many):
        prm, n = _abi.GroupMomentsParams(3, 2, 1, chunk), C.c_size_t()
        call = (lambda: lib.cs_b200_group_moments_parts_scratch_bytes(parts, 1, C.byref(prm), C.byref(n))) if many \
            else (lambda: lib.cs_b200_group_moments_scratch_bytes(C.byref(v), C.byref(prm), C.byref(n)))
        _abi.check(call(), "scratch")
        return n.value

    results = []
    for many in (False, True):
        assert need(0, many) > need(512, many) > need(2048, many)
        short = need(2048, many) - (4 if cols % 8 and not many else 0)
        for room in (need(0, many), need(512, many), need(2048, many), short):
            scratch = torch.full((room,), 0xff, dtype=torch.uint8, device="cuda")
            out = [torch.full((3, cols), -1.0, device="cuda") for _ in range(2)]
            status = torch.zeros(1, dtype=torch.int32, device="cuda")
            o, prm = _abi.GroupMomentsOut(*[dptr(t) for t in out]), _abi.GroupMomentsParams(3, 2, 1, 0)
            o.status = dptr(status)
            if many:
                ok = lib.cs_b200_group_moments_blocked_ell_parts(parts, 1, None, None, None, dptr(labels), C.byref(prm),
                                                                 C.byref(o), dptr(scratch), room, stream_handle())
            else:
                ok = lib.cs_b200_group_moments_blocked_ell(C.byref(v), None, None, dptr(labels), C.byref(prm),
                                                           C.byref(o), dptr(scratch), room, stream_handle())
            _abi.check(ok, "moments")
            results.append(torch.stack(out).cpu().numpy())
    for r in results[1:]:
        assert np.array_equal(r, results[0])  # whole counts: exact
