"""The calls a user of this framework makes, as measurable cases.

A case names a sparse matrix (a seeded synthetic graph or mesh, made on the
GPU), the width of the dense operand and the call: the products of the drop-in
module and of the tuned interface, a GCN layer, a training step, a batch of
sampled subgraphs, the ME-TCF conversion and the CSR relabelling. ``listed``
holds the fixed cases, ``draw`` makes further ones of the same ranges.

Matrix families (those of the benchmark configurations and the cost model's
training set): R-MAT graphs (symmetrised, self-loops, GCN-normalised values),
uniform random graphs (directed), block-diagonal clustered graphs with 5 %
off-block noise, the 27-point stencil, and Zipf-degree subgraphs for batches.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "dtc-spmm_asplos24_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

FORMS = ("tf32", "bf16x2x3", "split24x3", "split24x4", "bf16", "fp8")


def listed():
    return [
        # the smallest call: one product on a 4096-node sampled subgraph, hidden width 32
        dict(name="window_small_n32", kind="spmm", family="uniform", rows=4096, degree=8, N=32,
             call="window"),
        # a GCN layer (dense transform, aggregation, bias, ReLU) on a mini-batch subgraph whose
        # row count is no multiple of anything
        dict(name="layer_subgraph", kind="layer", family="uniform", rows=20011, degree=12, K=100,
             N=64),
        # the output layer of node classification: as many columns as classes, an odd number
        dict(name="classes_n41", kind="spmm", family="rmat", scale=17, degree=16, N=41,
             call="window"),
        # full-graph aggregation on a power-law graph, drop-in strict-balance call
        dict(name="balance_rmat20_n128", kind="spmm", family="rmat", scale=20, degree=16, N=128,
             call="balance"),
        # the same graph through the tuned interface within 1e-5: pack the fresh B, multiply
        dict(name="tuned_rmat20_n128", kind="spmm", family="rmat", scale=20, degree=16, N=128,
             call="tuned", form="bf16x2x3", H=32, W=8, mode=0, waves=64, ntile=0, pack=True),
        # the largest: a structured mesh, 2,000,376 rows, wide operand, tuned within 1e-5
        dict(name="tuned_stencil_n256", kind="spmm", family="stencil", n=126, N=256,
             call="tuned", form="bf16x2x3", H=32, W=8, mode=0, waves=32, ntile=2, pack=True),
        # full-batch training of one aggregation: forward with bias, gradient through A^T
        dict(name="train_directed_n64", kind="train", family="uniform", rows=250007, degree=16,
             N=64),
        # 128 sampled subgraphs of very uneven size, each with its own fresh features
        dict(name="batch_zipf_n64", kind="batch", count=128, rows_lo=256, rows_hi=65536, N=64),
        # low-precision inference with features packed once, wide operand, clustered graph
        dict(name="bf16_clustered_n512", kind="spmm", family="clustered", rows=131072, block=512,
             degree=32, N=512, call="tuned", form="bf16", H=16, W=8, mode=1, waves=16, ntile=0,
             pack=False),
        # preparing a full graph: CSR with values to ME-TCF
        dict(name="convert_rmat20", kind="convert", family="rmat", scale=20, degree=16, H=16, W=8,
             call="tuned"),
        # preparing a mini-batch subgraph, drop-in call
        dict(name="convert_subgraph", kind="convert", family="uniform", rows=20011, degree=12,
             H=16, W=8, call="dropin"),
        # the backward operand of a full graph: A^T as canonical CSR
        dict(name="transpose_rmat19", kind="relabel", family="rmat", scale=19, degree=16,
             op="transpose"),
    ]


# ------------------------------------------------------------------- drawing
def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_matrix(rng, hi):
    """A matrix of up to about `hi` nonzeros: small ones as likely as large ones."""
    family = rng.choice(("rmat", "uniform", "uniform", "clustered", "stencil"))
    nnz = _log(rng, 30000, hi)
    if family == "rmat":
        degree = rng.randint(4, 16)
        scale = int(round(math.log2(nnz / (2 * degree))))
        return dict(family=family, scale=max(11, min(20, scale)), degree=degree)
    if family == "stencil":
        return dict(family=family, n=max(11, min(100, int(round((nnz / 27) ** (1 / 3))))))
    degree = rng.randint(4, 64)
    rows = max(1501, min(1 << 20, nnz // degree)) + rng.randint(0, 15)
    if family == "uniform":
        return dict(family=family, rows=rows, degree=degree)
    return dict(family=family, rows=rows, degree=degree,
                block=1 << rng.randint(max(6, degree.bit_length() + 1), 12))


def draw(rng):
    kind = rng.choice(("spmm",) * 6 + ("layer", "train", "batch", "convert", "convert", "relabel"))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(16, 128), rows_lo=_log(rng, 128, 512),
                    rows_hi=_log(rng, 4096, 65536), N=rng.choice((16, 32, 64, 100, 128)))
    if kind == "convert":
        H, W = rng.choice(((16, 8), (16, 8), (32, 8), (16, 16)))
        return dict(kind=kind, H=H, W=W, call=rng.choice(("dropin", "tuned")),
                    **_draw_matrix(rng, 32000000))
    if kind == "relabel":
        return dict(kind=kind, op=rng.choice(("transpose", "permute")),
                    **_draw_matrix(rng, 32000000))
    mat = _draw_matrix(rng, 32000000)
    nnz, rows = _sizes(dict(mat))
    widths = [n for n in (8, 16, 32, 40, 41, 47, 64, 96, 100, 128, 200, 256, 384, 512)
              if nnz * n <= 5e9 and rows * n <= 1.4e8]
    N = rng.choice(widths or [8])
    if kind == "layer":
        return dict(kind=kind, K=rng.choice((32, 100, 128, 300)), N=N + N % 4 * 3, **mat)
    if kind == "train":
        return dict(kind=kind, N=N, **mat)
    call = rng.choice(("window", "balance", "tuned", "tuned"))
    if call != "tuned":
        return dict(kind=kind, N=N, call=call, **mat)
    form = rng.choice(("tf32", "tf32", "bf16x2x3", "bf16x2x3", "split24x3", "split24x4", "bf16",
                       "fp8"))
    unit = 4 if form == "tf32" else 16
    H, W = rng.choice(((16, 8), (32, 8), (16, 16)))
    mode = rng.randint(0, 1)
    return dict(kind=kind, N=(N + unit - 1) // unit * unit, call=call, form=form, H=H, W=W,
                mode=mode, waves=1 << rng.randint(0, 6 if mode == 0 else 4),
                ntile=rng.choice((0, 0, 1, 2)), pack=rng.random() < 0.5, **mat)


# ------------------------------------------------------------------ matrices
def _sizes(case):
    """(expected nonzeros, rows) of a case's matrix."""
    f = case["family"]
    if f == "rmat":
        rows = 1 << case["scale"]
        return int(0.92 * (2 * case["degree"] + 1) * rows), rows
    if f == "stencil":
        return (3 * case["n"] - 2) ** 3, case["n"] ** 3
    return case["rows"] * case["degree"], case["rows"]


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _csr(row, col, rows):
    """Distinct (row, col) pairs as CSR: int32 row pointer and columns, sorted."""
    key = torch.unique(row * rows + col)
    row = torch.div(key, rows, rounding_mode="floor")
    rowptr = torch.zeros(rows + 1, dtype=torch.int64, device="cuda")
    rowptr[1:] = torch.bincount(row, minlength=rows).cumsum(0)
    return rowptr.to(torch.int32), (key - row * rows).to(torch.int32), row


def _matrix(case, g):
    """(rowptr, col, val) on the device."""
    f = case["family"]
    rand = lambda n: torch.rand(n, generator=g, device="cuda")  # noqa: E731
    randint = lambda hi, n: torch.randint(hi, (n,), generator=g, device="cuda")  # noqa: E731
    if f == "rmat":
        scale, rows = case["scale"], 1 << case["scale"]
        n = case["degree"] * rows
        u = torch.zeros(n, dtype=torch.int64, device="cuda")
        v = torch.zeros(n, dtype=torch.int64, device="cuda")
        for _ in range(scale):  # quadrants with (a, b, c, d) = (0.57, 0.19, 0.19, 0.05)
            x = rand(n)
            u = 2 * u + (x >= 0.76)
            v = 2 * v + (((x >= 0.57) & (x < 0.76)) | (x >= 0.95))
        i = torch.arange(rows, device="cuda")
        rowptr, col, row = _csr(torch.cat((u, v, i)), torch.cat((v, u, i)), rows)
        deg = (rowptr[1:] - rowptr[:-1]).double()
        val = (deg[row] * deg[col.long()]).rsqrt().float()
        return rowptr, col, val
    if f == "stencil":
        n = case["n"]
        rows = n ** 3
        i = torch.arange(rows, dtype=torch.int32, device="cuda")
        z, y, x = i // (n * n), i // n % n, i % n
        d = torch.arange(-1, 2, dtype=torch.int32, device="cuda")
        dz, dy, dx = (t.reshape(-1) for t in torch.meshgrid(d, d, d, indexing="ij"))
        ok = torch.ones((rows, 27), dtype=torch.bool, device="cuda")
        for p, q in ((z, dz), (y, dy), (x, dx)):
            s = p[:, None] + q
            ok &= (s >= 0) & (s < n)
        col = i[:, None] + (dz * n + dy) * n + dx
        val = torch.randn((rows, 27), generator=g, device="cuda") * ok
        val[:, 13] = 0
        val[:, 13] = 27 + val.sum(1).abs()
        rowptr = torch.zeros(rows + 1, dtype=torch.int64, device="cuda")
        rowptr[1:] = ok.sum(1).cumsum(0)
        return rowptr.to(torch.int32), col[ok], val[ok]
    rows = case["rows"]
    if f == "uniform":
        deg = torch.poisson(torch.full((rows,), float(case["degree"]), device="cuda"),
                            generator=g).long()
    else:
        deg = torch.full((rows,), case["degree"], dtype=torch.int64, device="cuda")
    row = torch.repeat_interleave(torch.arange(rows, device="cuda"), deg)
    n = row.numel()
    col = randint(rows, n)
    if f == "clustered":
        first = row // case["block"] * case["block"]
        width = (rows - first).clamp(max=case["block"])
        inside = first + (rand(n).double() * width).long().clamp(max=case["block"] - 1)
        col = torch.where(rand(n) < 0.05, col, torch.minimum(inside, first + width - 1))
    rowptr, col, _ = _csr(row, col, rows)
    return rowptr, col, 2 * rand(col.numel()) - 1


def _shuffled(rowptr, col, val, g):
    """The matrix with its nodes renumbered in whole groups of 32: other arrays for each
    generator, with the sizes of every array of the conversion kept (no group, and so no row
    window, changes its number of nonzeros or distinct columns)."""
    rows = rowptr.numel() - 1
    i = torch.arange(rows, device="cuda")
    order = torch.randperm(rows // 32, generator=g, device="cuda")
    at = torch.empty(rows // 32 + 1, dtype=torch.int64, device="cuda")
    at[order] = torch.arange(rows // 32, device="cuda")
    at[-1] = rows // 32  # a last group of fewer rows stays where it is
    new = at[i // 32] * 32 + i % 32
    row = torch.repeat_interleave(new, rowptr.diff().long())
    rowptr, col, _ = _csr(row, new[col.long()], rows)
    return rowptr, col, val[torch.randperm(val.numel(), generator=g, device="cuda")]


def _zipf_batch(case, seed):
    """Square subgraphs on the host (sampled by the user's data loader): log-uniform row counts
    (the case's own), Zipf(2.1) degrees of at most 2000, row-normalised values."""
    from dtc_b200 import gen
    lo, hi, n = case["rows_lo"], case["rows_hi"], case["count"]
    rows = np.exp(np.random.default_rng(n).uniform(np.log(lo), np.log(hi), n)).astype(np.int64)
    rng = np.random.default_rng(seed)
    cdf = np.cumsum(np.arange(1, 2001, dtype=np.float64) ** -2.1)
    mats = []
    for m in rows.tolist():
        deg = np.minimum(1 + np.searchsorted(cdf / cdf[-1], rng.random(m)), m)
        row = np.repeat(np.arange(m, dtype=np.int64), deg)
        key = np.unique(row * m + rng.integers(0, m, row.size))
        row, col = key // m, (key % m).astype(np.int32)
        rowptr = np.zeros(m + 1, np.int32)
        rowptr[1:] = np.cumsum(np.bincount(row, minlength=m))
        val = rng.random(col.size).astype(np.float32) + np.float32(1e-3)
        val /= np.bincount(row, val, m).astype(np.float32)[row]
        mats.append(gen.CSR(rowptr, col, val, m, m))
    return mats


# ------------------------------------------------------------------- running
def _inputs(case, seed):
    """Everything the seed decides: the matrix and the dense operands."""
    g = _gen(seed)
    randn = lambda *s: torch.randn(s, generator=g, device="cuda")  # noqa: E731
    kind = case["kind"]
    if kind == "batch":
        mats = _zipf_batch(case, seed)
        return dict(mats=mats, Bs=[randn(m.M, case["N"]) for m in mats])
    if kind in ("convert", "relabel"):
        rowptr, col, val = _shuffled(*_matrix(case, _gen(1)), g)
    else:
        rowptr, col, val = _matrix(case, g)
    d = dict(rowptr=rowptr, col=col, val=val, M=rowptr.numel() - 1)
    if kind == "spmm":
        d["B"] = randn(d["M"], case["N"])
    elif kind == "layer":
        d["X"] = randn(d["M"], case["K"])
        d["Wt"] = randn(case["K"], case["N"]) / math.sqrt(case["K"])
        d["bias"] = randn(case["N"])
    elif kind == "train":
        d["X"], d["G"] = randn(d["M"], case["N"]), randn(d["M"], case["N"])
        d["bias"] = randn(case["N"])
    elif kind == "relabel":
        d["perm"] = torch.randperm(d["M"], generator=g, device="cuda").to(torch.int32)
    return d


def prepare(case, seed):
    from dtc_b200 import metcf, tune
    from dtc_b200.batched import BatchedSpMM
    kind = case["kind"]
    s = _inputs(case, seed)
    s["case"] = case
    if kind == "batch":
        s["plan"] = BatchedSpMM(s.pop("mats"), case["N"], mode=0)
        return s
    if kind == "convert":
        if case["call"] == "dropin":  # the caller's in-place outputs
            i32 = dict(dtype=torch.int32, device="cuda")
            nnz = s["col"].numel()
            s["bp"] = torch.zeros((s["M"] + case["H"] - 1) // case["H"], **i32)
            s["e2c"], s["e2r"] = torch.zeros(nnz, **i32), torch.zeros(nnz, **i32)
        return s
    if kind == "relabel":
        return s
    csr = (s.pop("rowptr"), s.pop("col"), s.pop("val"))
    s["m"] = metcf.convert(*csr[:2], s["M"], H=case.get("H", 16), W=case.get("W", 8),
                           values=csr[2])
    if kind == "train":
        rp, co, vo = metcf.transpose_csr(*csr, s["M"])
        s["mT"] = metcf.convert(rp, co, s["M"], values=vo)
    if case.get("call") == "tuned":
        s["fmt"], s["precision"] = tune.FORMS[case["form"]][:2]
        sms = torch.cuda.get_device_properties(0).multi_processor_count
        s["grid"] = case["waves"] * sms
        wsb = metcf.spmm_ex_workspace_bytes(s["m"], case["N"], case["mode"], s["grid"])
        s["ws"] = torch.empty(max(wsb, 1), dtype=torch.uint8, device="cuda")
        if case["form"] == "tf32":
            s["planes"] = [s["B"]]
        elif not case["pack"]:
            s["planes"] = metcf.pack_b(s.pop("B"), s["fmt"])
    return s


def run(s):
    import DTCSpMM
    from dtc_b200 import metcf
    case, kind = s["case"], s["case"]["kind"]
    if kind == "batch":
        s["plan"].load(s["Bs"])
        return s["plan"].run()
    if kind == "convert":
        H, W = case["H"], case["W"]
        if case["call"] == "dropin":
            out = DTCSpMM.preprocess_gpu(s["col"], s["rowptr"], s["M"], H, W, s["bp"], s["e2c"],
                                         s["e2r"])
            return list(out) + [s["bp"], s["e2c"], s["e2r"]]
        m = metcf.convert(s["rowptr"], s["col"], s["M"], H=H, W=W, values=s["val"])
        return dict(rwo=m.RowWindowOffset, rowid=m.TCblockRowid, tile=m.TCblocktileId,
                    toff=m.TCblockoffset, s2x=m.SparseAToX, bp=m.blockPartition,
                    e2c=m.edgeToColumn, e2r=m.edgeToRow, T=m.T, values=m.TCvalues)
    if kind == "relabel":
        if case["op"] == "transpose":
            return metcf.transpose_csr(s["rowptr"], s["col"], s["val"], s["M"])
        return metcf.permute_csr(s["rowptr"], s["col"], s["val"], s["perm"])
    m = s["m"]
    if kind == "layer":
        return metcf.gcn_layer(m, s["X"], s["Wt"], bias=s["bias"], relu=True)
    if kind == "train":
        mT = s["mT"]
        if case["N"] % 4 == 0:
            out = DTCSpMM.DTCSpMM_gcn(s["X"], m.RowWindowOffset, m.TCblocktileId, m.TCblockoffset,
                                      m.SparseAToX, m.M, m.nnz, values=m.TCvalues,
                                      bias=s["bias"])[0]
        else:  # the fused epilogue takes widths that are multiples of 4
            out = metcf.spmm(m, s["X"]) + s["bias"]
        grad = DTCSpMM.run_DTCSpMM_balance(s["G"], mT.TCblockRowid, mT.TCblocktileId,
                                           mT.TCblockoffset, mT.SparseAToX, m.M, "float4_split",
                                           values=mT.TCvalues)[0]
        return out, grad
    if case["call"] == "window":
        return DTCSpMM.run_DTCSpMM(s["B"], m.RowWindowOffset, m.TCblocktileId, m.TCblockoffset,
                                   m.SparseAToX, m.M, m.nnz, "float4_split", values=m.TCvalues)
    if case["call"] == "balance":
        return DTCSpMM.run_DTCSpMM_balance(s["B"], m.TCblockRowid, m.TCblocktileId,
                                           m.TCblockoffset, m.SparseAToX, m.M, "float4_split",
                                           values=m.TCvalues)
    planes = s["planes"] if "planes" in s else metcf.pack_b(s["B"], s["fmt"])
    return metcf.spmm_ex(m, planes, s["fmt"], case["N"], s["precision"], mode=case["mode"],
                         grid=s["grid"], workspace=s["ws"], ntile=case["ntile"])


def work(case):
    kind = case["kind"]
    if kind == "batch":
        lo, hi = case["rows_lo"], case["rows_hi"]
        rows = case["count"] * (hi - lo) / math.log(hi / lo)
        nnz = 3.9 * rows
    else:
        nnz, rows = _sizes(case)
    if kind == "convert":  # CSR in; ranks, rows, tile ids, gathered columns, offsets (values) out
        blocks = nnz / 8
        val = 8 if case["call"] == "tuned" else 0
        return dict(bytes=nnz * (4 + 9 + val) + blocks * (8 + 4 * case["W"]) + rows * 5,
                    flops=0)
    if kind == "relabel":
        return dict(bytes=nnz * 16 + rows * 8, flops=0)
    N = case["N"]
    # one product: tile ids, values and gathered columns of A, every B row once, C once
    eb = dict(tf32=4, bf16x2x3=4, split24x3=3, split24x4=3, bf16=2, fp8=1)[case.get("form", "tf32")]
    one = nnz * (1 + 4 + 4) + rows * N * (eb + 4)
    if kind == "layer":
        K = case["K"]
        return dict(bytes=one - rows * N * eb + rows * K * 4 + K * N * 4,
                    flops=2 * nnz * N + 2 * rows * K * N)
    if kind == "train":
        return dict(bytes=2 * one, flops=4 * nnz * N)
    if case.get("pack"):
        one += rows * N * 4 - rows * N * eb  # fp32 B is what comes in
    return dict(bytes=one, flops=2 * nnz * N)


# --------------------------------------------------------------- 64-bit truth
def _product(rowptr, col, val, B):
    M = rowptr.numel() - 1
    A = torch.sparse_csr_tensor(rowptr.long(), col.long(), val.double(), (M, B.shape[0]),
                                device="cuda")
    return A @ B.double()


def exact(case, seed):
    s = _inputs(case, seed)
    kind = case["kind"]
    if kind == "batch":
        outs = []
        for m, B in zip(s["mats"], s["Bs"]):
            dev = [torch.from_numpy(x).cuda() for x in (m.rowptr, m.col, m.val)]
            outs.append(torch.nn.functional.pad(_product(*dev, B), (0, 0, 0, -m.M % 16)))
        return torch.cat(outs)
    row = torch.repeat_interleave(torch.arange(s["M"], device="cuda"),
                                  s["rowptr"].diff().long())
    col = s["col"].long()
    if kind == "convert":
        if case["call"] == "dropin":
            return None  # whole numbers only
        win = torch.div(row, case["H"], rounding_mode="floor")
        pair, at = torch.unique(win * s["M"] + col, return_inverse=True)
        w = torch.div(pair, s["M"], rounding_mode="floor")
        first = torch.searchsorted(w, torch.arange(int(w[-1]) + 2, device="cuda"))
        block = win * s["M"] + torch.div(at - first[win], case["W"], rounding_mode="floor")
        order = torch.sort(block, stable=True).indices
        return dict(rwo=None, rowid=None, tile=None, toff=None, s2x=None, bp=None, e2c=None,
                    e2r=None, T=None, values=s["val"][order].double())
    if kind == "relabel":
        if case["op"] == "transpose":
            key = col * s["M"] + row
        else:
            inv = torch.empty_like(s["perm"], dtype=torch.int64)
            inv[s["perm"].long()] = torch.arange(s["M"], device="cuda")
            key = inv[row] * s["M"] + inv[col]
        return None, None, s["val"][torch.sort(key).indices].double()
    csr = (s["rowptr"], s["col"], s["val"])
    if kind == "layer":
        XW = s["X"].double() @ s["Wt"].double()
        return torch.relu(_product(*csr, XW) + s["bias"].double())
    if kind == "train":
        order = torch.sort(col * s["M"] + row).indices
        rp = torch.zeros(s["M"] + 1, dtype=torch.int64, device="cuda")
        rp[1:] = torch.bincount(col, minlength=s["M"]).cumsum(0)
        return (_product(*csr, s["X"]) + s["bias"].double(),
                _product(rp, row[order], s["val"][order], s["G"]))
    C = _product(*csr, s["B"])
    return C if case["call"] == "tuned" else [C]
