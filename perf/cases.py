"""The calls that programs built on this library make, as cases to time.

A case names one public entry point (``op``) and the matrix it is called on: cell x gene
count matrices of the synthetic generator (row sizes lognormal, gene popularity Zipf,
zero-truncated negative-binomial counts), from the 8,192 x 2,000 conversion matrix that the
tests use up to the 500,000 x 32,768 partition of the benchmark's grouped reduction, and
the forms that a program holds between the calls: CSR, COO in arrival order, Blocked-ELL,
Sliced-ELL.

``scaled`` values are counts times 0.731 rounded to fp16 (normalised counts, not integers);
``counts`` are whole numbers.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from cellshard_b200 import _abi, runtime, synth
from cellshard_b200.batch import BatchSlicedConverter
from cellshard_b200.device import (
    CSR,
    blocked_ell_from_coo,
    blocked_ell_from_csr,
    bucketed_sliced_ell,
    ptr,
    sliced_ell_from_csr,
    stream_handle,
    transpose,
    u32,
)


def listed():
    return [
        # The grouped reduction of the benchmark: per-group per-gene sums, moments of the kept
        # cells of one resident partition, buffers and the column-block index held by the caller.
        dict(name="moments_partition", op="moments", rows=500_000, cols=32_768, density=0.04, block=16, groups=64,
             row_keep=0.7, feature_keep=0.61, values="counts", resident=True),
        # The same question asked once of a small matrix (a notebook, a test): nothing held, so
        # allocation, the index and the launches count.
        dict(name="moments_small", op="moments", rows=8_192, cols=2_000, density=0.06, block=16, groups=8,
             row_keep=0.7, feature_keep=0.61, values="scaled", resident=False),
        # Per-cell quality control over the staged execution format: totals, detected genes,
        # maxima and gene-set shares.
        dict(name="reduce_blocked", op="reduce", form="blocked", rows=150_003, cols=32_768, density=0.04, block=16,
             groups=8, row_keep=0.7, feature_keep=0.6, values="counts"),
        # The same over CSR with many gene sets and normalised values, every cell kept.
        dict(name="reduce_csr", op="reduce", form="csr", rows=262_144, cols=20_011, density=0.05, block=0, groups=24,
             row_keep=1.0, feature_keep=0.6, values="scaled"),
        # Ingest of one small partition into the execution format: latency.
        dict(name="to_blocked_small", op="to_blocked", rows=8_192, cols=2_000, density=0.06, block=16),
        # Ingest of a large, ragged one: bandwidth.
        dict(name="to_blocked_large", op="to_blocked", rows=131_071, cols=32_768, density=0.04, block=16),
        # A shard of uneven partitions to Sliced-ELL with the slice height chosen and the row
        # plan made, one launch.
        dict(name="to_sliced_batch", op="to_sliced_batch", rows=400_000, cols=32_768, density=0.025, parts=12),
        # Cell-major to gene-major.
        dict(name="transpose_large", op="transpose", rows=300_000, cols=32_768, density=0.04),
        # Filter cells and genes of a staged partition, order the rows by size, rebuild.
        dict(name="repack", op="repack", rows=120_000, cols=32_768, density=0.04, block=16, row_keep=0.7,
             feature_keep=0.6, buckets=64),
        # Entries in arrival order (not row by row) into the execution format.
        dict(name="coo_shuffled", op="coo", rows=100_000, cols=32_768, density=0.04, block=16, shuffled=True),
        # Entries of a small upload.
        dict(name="coo_small", op="coo", rows=20_011, cols=5_003, density=0.03, block=16, shuffled=True),
        # Execution buckets of a Sliced-ELL partition, the bucket count chosen.
        dict(name="bucket_sliced", op="bucket_sliced", rows=250_007, cols=32_768, density=0.03, slice=32, buckets=0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the listed kinds: 2,000 cells up to the listed sizes, 1,000 to 33,000 genes,
    1 to 6 % density, the options that each entry point takes."""
    op = rng.choice(["moments", "reduce", "to_blocked", "to_sliced_batch", "transpose", "repack", "coo",
                     "bucket_sliced"])
    cols = _log(rng, 1_000, 33_000)
    density = rng.uniform(0.01, 0.06)
    top = {"moments": 300_000, "reduce": 250_000, "to_blocked": 131_000, "to_sliced_batch": 400_000,
           "transpose": 300_000, "repack": 110_000, "coo": 100_000, "bucket_sliced": 250_000}[op]
    rows = _log(rng, 2_000, top)
    # no more entries than the listed case of the kind
    most = {"to_sliced_batch": 320e6, "transpose": 390e6, "coo": 130e6, "bucket_sliced": 240e6}.get(op, 260e6)
    density = round(min(density, most / (rows * cols)), 5)
    c = dict(op=op, rows=rows, cols=cols, density=density)
    block = rng.choice([8, 16, 16, 32])
    values = rng.choice(["counts", "scaled"])
    keep = dict(row_keep=rng.choice([0.3, 0.7, 1.0]), feature_keep=round(rng.uniform(0.1, 1.0), 3))
    if op == "moments":
        c.update(block=block, groups=_log(rng, 2, 256), values=values, resident=rng.random() < 0.5, **keep)
    elif op == "reduce":
        form = rng.choice(["blocked", "sliced", "csr"])
        c.update(form=form, block=block if form == "blocked" else 0, groups=rng.randint(1, 32), values=values, **keep)
        if form == "sliced":
            c["slice"] = rng.choice([16, 32, 64])
    elif op == "to_blocked":
        c.update(block=block)
    elif op == "to_sliced_batch":
        c.update(parts=rng.randint(3, 12))
    elif op == "repack":
        c.update(block=block, buckets=rng.choice([16, 64]), **keep)
    elif op == "coo":
        c.update(block=block, shuffled=rng.random() < 0.75)
    elif op == "bucket_sliced":
        c.update(slice=rng.choice([16, 32, 64]), buckets=rng.choice([0, 4, 8]))
    return c


GROUP = 64  # rows that stay together: every slice height and row-block size divides it
BLOCK = 32  # columns that stay together: every block size divides it


def _columns(case, seed):
    """New column of each column of the case's base matrix: its 32-column blocks in another order."""
    cols = case["cols"]
    move = np.arange(cols)
    full = cols // BLOCK
    order = np.random.default_rng(seed + 3).permutation(full)
    move[:full * BLOCK] = (order[:, None] * BLOCK + np.arange(BLOCK)).reshape(-1)
    return move


def _csr(case, seed):
    """The case's matrix for one seed.  The seed deals the column blocks, the 64-row groups and
    the values anew; how many entries the rows and the row blocks hold is the case's own, so the
    results of two seeds have the same sizes."""
    spec = synth.MatrixSpec(case["rows"], case["cols"], case["density"] * case["cols"], 1, max(1, case["cols"] // 2))
    _n, rp, col_cdf, col_of_rank, val_cdf, _scale = synth.host_tables(spec)
    total = int(rp[-1])
    d_ptr, d_rank = u32(rp), u32(_columns(case, seed)[col_of_rank])
    d_cdf = torch.from_numpy(col_cdf.view(np.int64).copy()).cuda()
    d_vcdf = torch.from_numpy(val_cdf.view(np.int64).copy()).cuda()
    idx = torch.empty(total, dtype=torch.int32, device="cuda")
    val = torch.empty(total, dtype=torch.float16, device="cuda")
    _abi.check(_abi.load().cs_b200_synth_csr(spec.rows, spec.cols, ptr(d_ptr), ptr(d_cdf), ptr(d_rank), ptr(d_vcdf),
                                             len(val_cdf), None, spec.seed, ptr(idx), ptr(val), stream_handle()),
               "synth_csr")
    g = torch.Generator(device="cuda").manual_seed(seed + 11)
    if case["op"] != "repack":  # there, which rows share a block follows from the order of the sizes
        rows, full = case["rows"], case["rows"] // GROUP
        order = torch.randperm(full, generator=g, device="cuda")
        row = torch.cat([(order[:, None] * GROUP + torch.arange(GROUP, device="cuda")).reshape(-1),
                         torch.arange(full * GROUP, rows, device="cuda")])
        size = (d_ptr[1:] - d_ptr[:-1]).long()[row]
        new = torch.zeros(rows + 1, dtype=torch.int64, device="cuda")
        torch.cumsum(size, 0, out=new[1:])
        at = torch.repeat_interleave((d_ptr[:-1].long() & 0xFFFFFFFF)[row] - new[:-1], size)
        at += torch.arange(total, device="cuda")
        idx, d_ptr = idx[at], new.to(torch.int32)
        del at
    val = torch.roll(val, int(torch.randint(1, total, (1,), generator=g, device="cuda")))
    if case.get("values") == "scaled":
        val.mul_(0.731)
    return CSR(spec.rows, spec.cols, d_ptr, idx, val)


def _masks(case, seed):
    """(row_keep, feature_keep, labels, gene-set bits) on the device; a mask that keeps all is None."""
    rows, cols, groups = case["rows"], case["cols"], case.get("groups", 1)
    g = torch.Generator(device="cuda").manual_seed(seed + 17)
    rk = (torch.rand(rows, generator=g, device="cuda") < case["row_keep"]).to(torch.uint8)
    if case["op"] == "repack":  # the mask goes with its columns, and the rows stay
        fixed = torch.Generator(device="cuda").manual_seed(23)
        rk = (torch.rand(rows, generator=fixed, device="cuda") < case["row_keep"]).to(torch.uint8)
        fk = torch.empty(cols, dtype=torch.uint8, device="cuda")
        fk[torch.from_numpy(_columns(case, seed)).cuda()] = (
            torch.rand(cols, generator=fixed, device="cuda") < case["feature_keep"]).to(torch.uint8)
    else:
        fk = (torch.rand(cols, generator=g, device="cuda") < case["feature_keep"]).to(torch.uint8)
    labels = torch.randint(0, groups, (rows,), generator=g, device="cuda", dtype=torch.int32)
    # half of the genes are in no set, the others in each set with probability 1/2
    bits = torch.zeros(cols, dtype=torch.int64, device="cuda")
    for k in range(min(groups, 32)):
        bits |= (torch.rand(cols, generator=g, device="cuda") < 0.5).long() << k
    bits *= torch.rand(cols, generator=g, device="cuda") < 0.5
    bits = torch.where(bits >= 1 << 31, bits - (1 << 32), bits).to(torch.int32)
    return (None if case["row_keep"] >= 1.0 else rk), (None if case["feature_keep"] >= 1.0 else fk), labels, bits


FILTER = runtime.FilterParams(10.0, 5, 0.9, 0)


def prepare(case, seed):
    op = case["op"]
    csr = _csr(case, seed)
    st = {"op": op, "case": case}
    if op == "moments":
        bell = blocked_ell_from_csr(csr, case["block"])
        del csr
        st.update(bell=bell, index=None, ws=None, out=None)
        st["rk"], st["fk"], st["labels"], _ = _masks(case, seed)
        if case["resident"]:
            shape = (case["groups"], case["cols"])
            out = {k: torch.empty(shape, dtype=torch.float32, device="cuda") for k in ("sum", "sumsq", "mean", "var")}
            out["group_rows"] = torch.empty(case["groups"], dtype=torch.int32, device="cuda")
            out["status"] = torch.zeros(1, dtype=torch.int32, device="cuda")
            st.update(out=out, ws=runtime.MomentsWorkspace(), index=runtime.build_moments_index(bell, out["status"]))
    elif op == "reduce":
        if case["form"] == "blocked":
            src = blocked_ell_from_csr(csr, case["block"])
        elif case["form"] == "sliced":
            src = sliced_ell_from_csr(csr, case["slice"])
        else:
            src = csr
        st["src"] = src
        st["rk"], st["fk"], _, st["bits"] = _masks(case, seed)
    elif op in ("to_blocked", "transpose"):
        st["csr"] = csr
    elif op == "to_sliced_batch":
        r = np.random.default_rng(5)
        cut = np.sort(r.choice(np.arange(1, case["rows"] // GROUP), size=case["parts"] - 1, replace=False)) * GROUP
        cut = [0, *(int(x) for x in cut), case["rows"]]
        st_ptr = csr.ptr
        at = csr.ptr[torch.tensor(cut, device="cuda")].cpu().tolist()
        parts = [CSR(b - a, case["cols"], csr.ptr[a:b + 1] - p, csr.idx[p:q].clone(), csr.val[p:q].clone())
                 for a, b, p, q in zip(cut, cut[1:], at, at[1:])]
        del csr
        # room for every partition at the tallest slices, as arena_bound gives it for any order of the groups
        n = (st_ptr[1:] - st_ptr[:-1]).cpu().numpy().astype(np.float64)
        room = int(6 * max(_slots(n, h) for h in (16, 32, 64))) + case["rows"] + 4096 * case["parts"]
        conv = BatchSlicedConverter(parts, arena_bytes=room)
        conv.arena.zero_()  # the gaps between the blocks are compared too
        for o in conv.plan_out:
            for t in o.values():
                t.zero_()
        st["conv"] = conv
    elif op == "repack":
        st["bell"] = blocked_ell_from_csr(csr, case["block"])
        del csr
        st["rk"], st["fk"], _, _ = _masks(case, seed)
    elif op == "coo":
        row = torch.repeat_interleave(torch.arange(case["rows"], device="cuda", dtype=torch.int32),
                                      (csr.ptr[1:] - csr.ptr[:-1]).long())
        col, val = csr.idx, csr.val
        if case["shuffled"]:
            g = torch.Generator(device="cuda").manual_seed(seed + 29)
            order = torch.randperm(row.numel(), generator=g, device="cuda")
            row, col, val = row[order], col[order], val[order]
        st.update(row=row, col=col, val=val)
    elif op == "bucket_sliced":
        st["sell"] = sliced_ell_from_csr(csr, case["slice"])
        del csr
    return st


def _bits(t):
    """fp16 values that are only moved, as their bits."""
    return t.view(torch.int16)


def _bell(b):
    return {"ell_cols": b.ell_cols, "nnz": b.nnz, "bci": b.bci, "val": _bits(b.val)}


def _compressed(c):
    return {"ptr": c.ptr, "idx": c.idx, "val": _bits(c.val)}


def run(st):
    op, case = st["op"], st["case"]
    if op == "moments":
        return runtime.compute_sparse_group_moments(st["bell"], case["groups"], st["rk"], st["fk"], st["labels"],
                                                    workspace=st["ws"], out=st["out"], index=st["index"])
    if op == "reduce":
        return runtime.compute_sparse_group_reduce(st["src"], st["bits"], case["groups"], st["rk"], st["fk"], FILTER)
    if op == "to_blocked":
        return _bell(blocked_ell_from_csr(st["csr"], case["block"]))
    if op == "to_sliced_batch":
        conv = st["conv"]
        conv.run()
        results, deferred, err = conv.results()
        return {"arena": conv.arena.view(torch.int32), "plans": conv.plan_out,
                "counts": torch.tensor([deferred, err]), "slices": torch.tensor(
                    [[r.slice_rows, r.slice_count, r.total_slots] for r in results])}
    if op == "transpose":
        return _compressed(transpose(st["csr"]))
    if op == "repack":
        filtered, plan, rebuilt, bell, stats = runtime.build_repacked_blocked_ell(
            [st["bell"]], case["rows"], case["cols"], case["block"], case["buckets"], st["rk"], st["fk"])
        return {"filtered": _compressed(filtered), "plan": plan, "rebuilt": _compressed(rebuilt), "bell": _bell(bell),
                "kept": [stats["kept_rows"], stats["live_nnz"], stats["kept_row_slots"]]}
    if op == "coo":
        bell, counts, status, total = blocked_ell_from_coo(case["rows"], case["cols"], st["row"], st["col"], st["val"],
                                                           case["block"], case["cols"])
        return {"bell": _bell(bell), "counts": counts, "status": status, "total": total}
    b = bucketed_sliced_ell(st["sell"], case["buckets"])
    return {"plan": b.plan, "offsets": torch.tensor(b.segment_row_offsets), "to_canonical": b.exec_to_canonical_rows,
            "to_exec": b.canonical_to_exec_rows, "idx": b.idx, "val": _bits(b.val)}


def exact(case, seed):
    """The reductions' values in 64 bits; the other calls only move and count."""
    if case["op"] not in ("moments", "reduce"):
        return None
    csr = _csr(case, seed)
    rk, fk, labels, bits = _masks(case, seed)
    rows, cols, groups = case["rows"], case["cols"], case["groups"]
    dev = "cuda"
    rk = torch.ones(rows, dtype=torch.bool, device=dev) if rk is None else rk.bool()
    fk = torch.ones(cols, dtype=torch.bool, device=dev) if fk is None else fk.bool()
    start = csr.ptr.long()
    step = max(1, rows // max(1, csr.nnz // (1 << 26) + 1))

    def chunks():
        for a in range(0, rows, step):
            b = min(rows, a + step)
            p, q = int(start[a]), int(start[b])
            row = torch.repeat_interleave(torch.arange(a, b, device=dev), start[a + 1:b + 1] - start[a:b])
            col, val = csr.idx[p:q].long(), csr.val[p:q].double()
            ok = rk[row] & fk[col] & (val != 0)
            yield row[ok], col[ok], val[ok]

    if case["op"] == "moments":
        s = torch.zeros(groups * cols, dtype=torch.float64, device=dev)
        q = torch.zeros_like(s)
        for row, col, val in chunks():
            key = labels[row].long() * cols + col
            s.index_add_(0, key, val)
            q.index_add_(0, key, val * val)
        s, q = s.view(groups, cols), q.view(groups, cols)
        n = torch.bincount(labels[rk].long(), minlength=groups).double()[:, None]
        mean = torch.where(n > 0, s / n.clamp(min=1), torch.zeros_like(s))
        var = torch.where(n > 1, (q - s * s / n.clamp(min=1)) / (n - 1).clamp(min=1), torch.zeros_like(s))
        return {"sum": s, "sumsq": q, "mean": mean, "var": var, "group_rows": None, "status": None}
    total = torch.zeros(rows, dtype=torch.float64, device=dev)
    top = torch.zeros(rows, dtype=torch.float64, device=dev)
    sets = torch.zeros(rows, groups, dtype=torch.float64, device=dev)
    for row, col, val in chunks():
        total.index_add_(0, row, val)
        top.scatter_reduce_(0, row, val, "amax")
        m = bits[col]
        for k in range(groups):
            sets[:, k].index_add_(0, row, torch.where((m >> k) & 1 == 1, val, torch.zeros_like(val)))
    t = total[:, None]
    share = torch.where(t > 0, 100.0 * sets / t.clamp(min=1e-300), torch.zeros_like(sets))
    return {"row_totals": total, "detected_features": None, "max_values": top, "row_keep": None,
            "group_counts": sets.reshape(-1), "group_percentages": share.reshape(-1)}


def _sizes(case):
    """(row sizes, entries, padded columns of a Blocked-ELL row) that the case's matrix has, near enough."""
    rows, cols = case["rows"], case["cols"]
    n = synth.row_nnz(rows, case["density"] * cols, 0.6, 1, max(1, cols // 2), np.random.default_rng(1)).astype(np.float64)
    block = case.get("block") or 0
    padded = 0
    if block:
        # distinct block columns of the fullest row block: popularity Zipf(1.1), dealt over the columns
        whole = rows // block * block
        most = n[:whole].reshape(-1, block).sum(1).max() if whole else n.sum()
        p = np.arange(1, cols + 1, dtype=np.float64) ** -1.1
        p = np.random.default_rng(2).permutation(p / p.sum())
        nb = -(-cols // block)
        q = np.add.reduceat(p, np.arange(0, cols, block))
        # columns are drawn without replacement, so popular ones fill up: find the draws that give `most`
        k = min(most / block, 0.999 * cols)
        lo, hi = 0.0, 1e9
        for _ in range(60):
            mid = (lo + hi) / 2
            lo, hi = (mid, hi) if (1 - np.exp(-mid * p)).sum() < k else (lo, mid)
        padded = block * min(nb, float((1 - np.exp(-lo * block * q)).sum()) + 2)
    return n, float(n.sum()), padded


def work(case):
    """Each input read once (rows that the mask drops are not), each output written once."""
    rows, cols, op = case["rows"], case["cols"], case["op"]
    n, nnz, padded = _sizes(case)
    csr = 4.0 * (rows + 1) + 6.0 * nnz
    blocks = -(-rows // case["block"]) if case.get("block") else 0
    bell = rows * padded * 2.0 + (blocks * padded / case["block"] * 4.0 if blocks else 0.0)
    keep, fkeep = case.get("row_keep", 1.0), case.get("feature_keep", 1.0)
    flops = 0.0
    if op == "moments":
        nbytes = keep * bell + 5.0 * rows + cols + case["groups"] * cols * 16.0
        flops = 3.0 * keep * nnz
    elif op == "reduce":
        if case["form"] == "blocked":
            src = bell
        elif case["form"] == "sliced":
            src = 6.0 * _slots(n, case["slice"])
        else:
            src = csr
        nbytes = keep * src + rows + 5.0 * cols + rows * (13.0 + 8.0 * case["groups"])
        flops = keep * fkeep * nnz * (1 + case["groups"] / 4)
    elif op == "to_blocked":
        nbytes = csr + bell
    elif op == "transpose":
        nbytes = csr + 4.0 * (cols + 1) + 6.0 * nnz
    elif op == "to_sliced_batch":
        nbytes = csr + 6.0 * _slots(n, 16) + 12.0 * rows
    elif op == "repack":
        kept = keep * fkeep * nnz
        nbytes = keep * bell + 2 * (4.0 * (rows + 1) + 6.0 * kept) + 16.0 * rows + keep * bell
    elif op == "coo":
        nbytes = 10.0 * nnz + bell
    else:
        nbytes = 6.0 * _slots(n, case["slice"]) + 6.0 * nnz * 1.05 + 8.0 * rows
    return {"bytes": nbytes, "flops": flops}


def _slots(n, height):
    pad = np.zeros(-len(n) % height)
    return float(np.concatenate([n, pad]).reshape(-1, height).max(1).sum() * height)
