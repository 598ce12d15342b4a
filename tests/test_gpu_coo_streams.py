"""The COO plan is complete when it returns: its stream is idle, and the emit
runs on another stream, with and without a repeated (row, column)."""

import ctypes as C

import numpy as np
import pytest

from cases import np_u16, np_u32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,n,order,repeat", [
    (5_000, 2_000, 3_000_000, "shuffled", 0),    # any order of a row's entries
    (5_000, 2_000, 3_000_000, "shuffled", 3),    # repeats found by the shape pass: ordered again
    (5_000, 2_000, 3_000_000, "by rows", 0),     # no partition
    (2_097_153, 16, 300_000, "shuffled", 2),     # past the partition: two sorts
])
def test_plan_and_emit_on_two_streams(cuda, orc, rows, cols, n, order, repeat):
    import torch

    from cellshard_b200 import _abi

    rng = np.random.default_rng(rows + repeat)
    block = 16
    cell = np.unique(rng.integers(0, rows * cols, n))
    cell = rng.permutation(np.append(cell, cell[:repeat]))
    if order == "by rows":
        cell = np.sort(cell)
    row, col = (cell // cols).astype(np.uint32), (cell % cols).astype(np.uint32)
    val = rng.integers(1, 2000, len(cell)).astype(np.float16).view(np.uint16)
    dev = [torch.from_numpy(a.view(t).copy()).cuda() for a, t in ((row, np.int32), (col, np.int32), (val, np.float16))]
    lib = _abi.load()
    v = _abi.CooView()
    v.rows, v.cols, v.nnz = rows, cols, len(cell)
    v.rowIdx, v.colIdx, v.val = (t.data_ptr() for t in dev)
    nbytes, width, total = C.c_size_t(), C.c_uint32(), C.c_uint64()
    _abi.check(lib.cs_b200_coo_blocked_ell_scratch_bytes(len(cell), rows, cols, block, C.byref(nbytes)), "scratch")
    scratch = torch.empty(nbytes.value, dtype=torch.uint8, device="cuda")
    words = torch.zeros(3, dtype=torch.int64, device="cuda")
    plan_on, emit_on = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    _abi.check(lib.cs_b200_coo_blocked_ell_plan(C.byref(v), None, cols, block, scratch.data_ptr(), nbytes.value,
                                                C.byref(width), C.byref(total), words.data_ptr() + 16,
                                                plan_on.cuda_stream), "plan")
    assert plan_on.query()
    W, RB = width.value, (rows + block - 1) // block
    bci = torch.empty(max(RB * W, 1), dtype=torch.int32, device="cuda")
    out = torch.empty(rows * W * block, dtype=torch.float16, device="cuda")
    d = _abi.BlockedEllView(rows, cols, 0, block, W * block, bci.data_ptr(), out.data_ptr())
    _abi.check(lib.cs_b200_coo_blocked_ell_emit(C.byref(v), None, cols, scratch.data_ptr(), nbytes.value, C.byref(d),
                                                words.data_ptr(), emit_on.cuda_stream), "emit")
    torch.cuda.synchronize()
    ref = orc.blocked_ell_from_coo(rows, cols, row, col, val, block, None)
    assert W * block == ref["ell_cols"] and total.value == ref["total_blocks"]
    assert words.tolist() == [ref["nnz_host"], ref["nnz_gpu"], 0]
    assert np.array_equal(np_u32(bci), ref["bci"]) and np.array_equal(np_u16(out), ref["val"])
