"""Performance cases of the SpMV library, through its public Python entry points.

Four kinds of work, each with the arrays that a user's program keeps between
calls (matrix, plan, vectors) made on the GPU from a seed:

* ``spmv``     one ``sparse_mv`` / ``sparse_mv_mixed`` on a built format;
* ``grad``     forward and backward of ``autograd.spmv`` (dx and dvalues);
* ``batched``  one ``SpMVBatch`` product over many uneven matrices, k
  right-hand sides;
* ``cg``       one conjugate-gradient solve.

``listed()`` gives the named cases, ``draw(rng)`` further ones of the same
ranges, ``prepare`` / ``run`` one state and one pass, ``work`` the bytes and
operations a pass cannot do without, ``exact`` the fp64 result from plain
torch operations.
"""
from __future__ import annotations

import math

import torch

import rvvlasparse_b200 as R
from rvvlasparse_b200 import autograd, batched, solvers

FORMATS = {"hcsr": R.spMtxHCSR, "sell": R.spMtxSELL_C_Sigma, "csr5": R.spMtxCSR5, "lav": R.spMtxLAV,
           "vnec": R.spMtxVNEC, "vhcc": R.spMtxVHCC, "cvr": R.spMtxCVR}
MIXED_FORMATS = ("crs", "hcsr", "csr5", "sell")
DTYPES = {"f64": torch.float64, "f32": torch.float32, "mixed": torch.float32, "mixed_bf16": torch.bfloat16}
CG_SHIFT = 0.5  # diagonal shift of the solver's Laplacian (an implicit time step)


# ------------------------------------------------------------------ cases


def _spmv(fmt, prec, matrix, n, **kw):
    return {"kind": "spmv", "format": fmt, "prec": prec, "matrix": matrix, "n": n, **kw}


def listed():
    return [
        # One product with a small 2-D Laplacian (256 x 256 grid) in the plain
        # CRS form: the smallest call, launch and host latency.
        {"name": "crs_f64_laplace256", **_spmv("crs", "f64", "laplace2d", 256)},
        # The headline matrix: 4M rows, lognormal row lengths, banded plus
        # random columns; the plain double-precision product.
        {"name": "crs_f64_powerlaw4M", **_spmv("crs", "f64", "powerlaw", 4194304)},
        # Mixed precision (fp32 values, compensated sums) on the 27-point
        # stencil of a 128^3 grid, the PDE matrix of the precision workload.
        {"name": "csr5_mixed_stencil128", **_spmv("csr5", "mixed", "stencil27", 128)},
        # The reference's own blocked format at its default block size, on an
        # irregular matrix whose size divides by no block or tile.
        {"name": "hcsr_f64_powerlaw1M", **_spmv("hcsr", "f64", "powerlaw", 1000003)},
        # Sliced ELL in single precision, default C and sigma, headline matrix.
        {"name": "sell_f32_powerlaw4M", **_spmv("sell", "f32", "powerlaw", 4194304)},
        # The vectorised formats of the reference on irregular matrices of
        # 1M to 2M rows, single and double precision.
        {"name": "lav_f64_powerlaw2M", **_spmv("lav", "f64", "powerlaw", 2097152)},
        {"name": "vhcc_f32_powerlaw2M", **_spmv("vhcc", "f32", "powerlaw", 1999993)},
        {"name": "cvr_f64_random1M", **_spmv("cvr", "f64", "random", 1048576, mean=19.0)},
        # A training step through the product: y, dvalues and dx on a random
        # pattern with 20M nonzeros in fp32.
        {"name": "grad_f32_random1M", "kind": "grad", "prec": "f32", "n": 1048576, "mean": 19.0},
        # Many independent matrices in one launch, plan tuned by the library:
        # one vector each, and a block of eight right-hand sides each.
        {"name": "batched_f32_256_k1", "kind": "batched", "prec": "f32", "count": 256, "n_lo": 1024, "n_hi": 65536,
         "k": 1, "tune": True},
        {"name": "batched_f32_256_k8", "kind": "batched", "prec": "f32", "count": 256, "n_lo": 1024, "n_hi": 65536,
         "k": 8, "tune": True},
        # A whole solve: CG on a shifted 2-D Laplacian, 2048 x 2048 grid, to
        # 1e-8.
        {"name": "cg_f64_laplace2048", "kind": "cg", "prec": "f64", "n": 2048},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: sizes log-uniform over the listed range, any format,
    precision and matrix family."""
    kind = rng.choice(["spmv"] * 7 + ["grad", "batched", "cg"])
    if kind == "spmv":
        fmt = rng.choice(["crs", "crs", "hcsr", "sell", "csr5", "lav", "vnec", "vhcc", "cvr"])
        prec = rng.choice(["f64", "f32", "mixed", "mixed_bf16"] if fmt in MIXED_FORMATS else ["f64", "f32"])
        matrix = rng.choice(["powerlaw", "powerlaw", "random", "stencil27", "laplace2d"])
        if matrix == "powerlaw":
            return _spmv(fmt, prec, matrix, _log_int(rng, 30000, 4194304 if fmt != "hcsr" else 2097152))
        if matrix == "random":
            return _spmv(fmt, prec, matrix, _log_int(rng, 30000, 1500000), mean=round(rng.uniform(4.0, 40.0), 2))
        if matrix == "stencil27":
            return _spmv(fmt, prec, matrix, _log_int(rng, 24, 128))
        return _spmv(fmt, prec, matrix, _log_int(rng, 181, 2048))
    if kind == "grad":
        return {"kind": "grad", "prec": rng.choice(["f32", "f64"]), "n": _log_int(rng, 30000, 1048576),
                "mean": round(rng.uniform(4.0, 30.0), 2)}
    if kind == "batched":
        return {"kind": "batched", "prec": rng.choice(["f32", "f32", "f64"]), "count": _log_int(rng, 16, 256),
                "n_lo": 1024, "n_hi": _log_int(rng, 4096, 65536), "k": rng.choice([1, 1, 4, 8]),
                "tune": rng.random() < 0.5}
    return {"kind": "cg", "prec": rng.choice(["f64", "f32"]), "n": _log_int(rng, 181, 2048)}


# ------------------------------------------------------------------ matrices


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _uniform(size, g, dtype=torch.float64):
    return torch.rand(size, generator=g, device="cuda", dtype=dtype).mul_(2).sub_(1)


def _rows_to_crs(m, n, row, col):
    """Sorted, duplicate-free CRS pattern of the entries (row, col)."""
    key = torch.sort(row * n + col).values
    keep = torch.ones_like(key, dtype=torch.bool)
    keep[1:] = key[1:] != key[:-1]
    key = key[keep]
    row, col = key // n, (key % n).to(torch.int32)
    Rst = torch.zeros(m + 1, dtype=torch.int64, device="cuda")
    Rst[1:] = torch.cumsum(torch.bincount(row, minlength=m), 0)
    return Rst.to(torch.int32), col


def _powerlaw(n, g):
    """Lognormal row lengths (mean 16, sigma 1.2, at most 4096), 70 % of the
    columns within +-1024 of the diagonal, the rest uniform."""
    z = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    ln = torch.exp(math.log(16.0) - 0.72 + 1.2 * z).round().clamp(1, min(4096, n)).long()
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), ln)
    nz = row.numel()
    near = row + torch.randint(-1024, 1025, (nz,), generator=g, device="cuda")
    far = torch.randint(0, n, (nz,), generator=g, device="cuda")
    band = torch.rand(nz, generator=g, device="cuda") < 0.7
    return _rows_to_crs(n, n, row, torch.where(band, near.clamp_(0, n - 1), far))


def _random(m, mean, g):
    """Geometric row lengths of the given mean in a random order, one column
    at random from each of the row's equal shares of the columns (distinct
    and sorted).  The lengths, and with them the number of nonzeros, are the
    same for every seed; their order and the columns are not."""
    fixed = _gen(m)
    u = torch.rand(m, generator=fixed, device="cuda", dtype=torch.float64).clamp_(min=1e-300)
    ln = (1 + torch.floor(torch.log(u) / math.log1p(-1.0 / mean))).long().clamp_(1, m)
    ln = ln[torch.randperm(m, generator=g, device="cuda")]
    Rst = torch.zeros(m + 1, dtype=torch.int64, device="cuda")
    Rst[1:] = torch.cumsum(ln, 0)
    row = torch.repeat_interleave(torch.arange(m, device="cuda"), ln)
    k = torch.arange(row.numel(), device="cuda") - Rst[row]
    lo, hi = k * m // ln[row], (k + 1) * m // ln[row]
    u = torch.rand(row.numel(), generator=g, device="cuda", dtype=torch.float64)
    col = torch.minimum(lo + (u * (hi - lo)).long(), hi - 1)
    return Rst.to(torch.int32), col.to(torch.int32)


def _stencil27(side):
    n = side ** 3
    i = torch.arange(n, device="cuda")
    z, y, x = i // (side * side), (i // side) % side, i % side
    cols = [(((z + dz) % side) * side + (y + dy) % side) * side + (x + dx) % side
            for dz in (-1, 0, 1) for dy in (-1, 0, 1) for dx in (-1, 0, 1)]
    col = torch.sort(torch.stack(cols, 1), 1).values.reshape(-1).to(torch.int32)
    return torch.arange(0, 27 * n + 1, 27, device="cuda", dtype=torch.int32), col


def _laplace2d(side):
    """Pattern and values of the 5-point Laplacian (4 on the diagonal, -1 off
    it, Dirichlet boundary)."""
    n = side * side
    i = torch.arange(n, device="cuda")
    r, c = i // side, i % side
    ok = torch.stack([r > 0, c > 0, torch.ones_like(r, dtype=torch.bool), c < side - 1, r < side - 1], 1)
    off = torch.tensor([-side, -1, 0, 1, side], device="cuda")
    col = (i[:, None] + off)[ok].to(torch.int32)
    Val = torch.tensor([-1.0, -1.0, 4.0, -1.0, -1.0], device="cuda", dtype=torch.float64).expand(n, 5)[ok]
    Rst = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    Rst[1:] = torch.cumsum(ok.sum(1), 0)
    return Rst.to(torch.int32), col, Val


def _matrix(case, g):
    """(n, Rst, Col, fp64 values) of an spmv case."""
    if case["matrix"] == "powerlaw":
        n = case["n"]
        Rst, Col = _powerlaw(n, g)
        Val = _uniform(Col.numel(), g)
    elif case["matrix"] == "random":
        n = case["n"]
        Rst, Col = _random(n, case["mean"], g)
        Val = torch.randn(Col.numel(), generator=g, device="cuda", dtype=torch.float64)
    elif case["matrix"] == "stencil27":
        n = case["n"] ** 3
        Rst, Col = _stencil27(case["n"])
        Val = 1.0 + 0.1 * torch.randn(Col.numel(), generator=g, device="cuda", dtype=torch.float64)
    else:
        n = case["n"] ** 2
        Rst, Col, Val = _laplace2d(case["n"])
    return n, Rst, Col, Val


def _crs(n, Rst, Col, Val):
    return R.spMtxCRS(n, n, int(Col.numel()), Rst, Col, Val)


def _row_of(Rst):
    m = Rst.numel() - 1
    return torch.repeat_interleave(torch.arange(m, device=Rst.device), torch.diff(Rst.long()))


def _batch_arrays(case, g):
    """All matrices of a batch in one set of arrays: sizes, first rows, row
    pointers over all of them, columns, values in the case's type.  Poisson
    row lengths, average nonzeros per row uniform in [4, 64], uniform
    columns."""
    count, lo, hi = case["count"], case["n_lo"], case["n_hi"]
    # the sizes are the same for every seed: a batch's cost is its case's
    fixed = torch.Generator()
    fixed.manual_seed(count * 1000003 + hi)
    ns = torch.exp(math.log(lo) + torch.rand(count, generator=fixed, dtype=torch.float64)
                   * math.log(hi / lo)).long()
    avg = 4.0 + 60.0 * torch.rand(count, generator=fixed, dtype=torch.float64)
    start = torch.zeros(count + 1, dtype=torch.int64)
    start[1:] = torch.cumsum(ns, 0)
    mat = torch.repeat_interleave(torch.arange(count), ns).cuda()
    nrow = ns.cuda()[mat]
    ln = torch.minimum(torch.poisson(avg.cuda()[mat], generator=g).long(), nrow)
    row = torch.repeat_interleave(torch.arange(mat.numel(), device="cuda"), ln)
    col = (torch.rand(row.numel(), generator=g, device="cuda", dtype=torch.float64) * nrow[row]).long()
    Rst, Col = _rows_to_crs(mat.numel(), int(ns.max()), row, col)
    Val = _uniform(Col.numel(), g, DTYPES[case["prec"]])
    return ns.tolist(), start.tolist(), Rst, Col, Val


# ------------------------------------------------------------------ prepare


def _inputs(case, seed):
    """The seeded inputs of a case before any library call."""
    g = _gen(seed)
    dt = DTYPES[case["prec"]]
    if case["kind"] == "spmv":
        n, Rst, Col, Val = _matrix(case, g)
        x = _uniform(n, g).to(torch.float64 if case["prec"] == "f64" else torch.float32)
        return {"n": n, "Rst": Rst, "Col": Col, "Val": Val.to(dt), "x": x}
    if case["kind"] == "grad":
        n = case["n"]
        Rst, Col = _random(n, case["mean"], g)
        v, x, u = (torch.randn(s, generator=g, device="cuda", dtype=dt) for s in (Col.numel(), n, n))
        return {"n": n, "Rst": Rst, "Col": Col, "Val": v, "x": x, "g": u}
    if case["kind"] == "batched":
        ns, start, Rst, Col, Val = _batch_arrays(case, g)
        X = _uniform(start[-1] * case["k"], g, dt)
        return {"ns": ns, "start": start, "Rst": Rst, "Col": Col, "Val": Val, "x": X}
    Rst, Col, Val = _laplace2d(case["n"])
    n = case["n"] ** 2
    Val = torch.where(Val > 0, Val + CG_SHIFT, Val).to(dt)
    return {"n": n, "Rst": Rst, "Col": Col, "Val": Val, "x": _uniform(n, g).to(dt)}


def prepare(case, seed):
    d = _inputs(case, seed)
    st = {"case": case}
    if case["kind"] == "spmv":
        fmt, prec = case["format"], case["prec"]
        n, val = d["n"], d["Val"]
        # bf16 storage is a rounded copy of the built fp32 matrix
        A = _crs(n, d["Rst"], d["Col"], val.float() if prec == "mixed_bf16" else val)
        if fmt != "crs":
            params = {"segment_len": n} if fmt == "lav" else {}  # x fits the L2: one column segment
            A = R.convert(FORMATS[fmt](), A, R.convertParams(**params))
        if prec == "mixed_bf16":
            A = A.astype(torch.bfloat16)
        st.update(A=A, x=d["x"], y=torch.zeros(n, dtype=d["x"].dtype, device="cuda"),
                  descr=R.sparse_matrix_descr(), mv=R.sparse_mv_mixed if prec.startswith("mixed") else R.sparse_mv)
    elif case["kind"] == "grad":
        pattern = autograd.CrsPattern(d["n"], d["n"], d["Rst"], d["Col"], d["Val"].dtype)
        st.update(pattern=pattern, values=d["Val"].requires_grad_(True), x=d["x"].requires_grad_(True), g=d["g"])
    elif case["kind"] == "batched":
        Rst, start = d["Rst"], d["start"]
        cut = Rst[torch.tensor(start, device="cuda")].tolist()
        mats = []
        for i, n in enumerate(d["ns"]):
            rst = Rst[start[i]:start[i + 1] + 1] - cut[i]
            mats.append(_crs(n, rst, d["Col"][cut[i]:cut[i + 1]].clone(), d["Val"][cut[i]:cut[i + 1]].clone()))
        B = batched.SpMVBatch(mats, k=case["k"], tune=case["tune"])
        st.update(B=B, X=d["x"], Y=torch.zeros(B.y_len, dtype=d["x"].dtype, device="cuda"))
    else:
        st.update(A=_crs(d["n"], d["Rst"], d["Col"], d["Val"]), b=d["x"],
                  rtol=1e-8 if case["prec"] == "f64" else 1e-5)
    return st


def run(st):
    kind = st["case"]["kind"]
    if kind == "spmv":
        status = st["mv"](R.SPARSE_OPERATION_NON_TRANSPOSE, 1.0, st["A"], st["descr"], st["x"], 0.0, st["y"])
        if status.code:
            raise RuntimeError(f"sparse_mv: status {status.code}")
        return st["y"]
    if kind == "grad":
        y = autograd.spmv(st["pattern"], st["values"], st["x"])
        dv, dx = torch.autograd.grad(y, (st["values"], st["x"]), st["g"])
        return {"y": y.detach(), "dvalues": dv, "dx": dx}
    if kind == "batched":
        code = st["B"].spmv(1.0, st["X"], 0.0, st["Y"])
        if code:
            raise RuntimeError(f"SpMVBatch.spmv: status {code}")
        return st["Y"]
    x, it, _ = solvers.cg(st["A"], st["b"], rtol=st["rtol"], max_iter=400, check_every=10)
    return {"x": x, "iterations": it}


# ------------------------------------------------------------------ work


def _shape(case):
    """(rows, nonzeros) of one pass, the nonzeros from the generators' means."""
    n = case["n"]
    if case.get("matrix") == "stencil27":
        return n ** 3, 27 * n ** 3
    if case["kind"] == "cg" or case.get("matrix") == "laplace2d":
        return n * n, 5 * n * n - 4 * n
    return n, int(n * (case["mean"] if "mean" in case else 16.0))


def work(case):
    vb = {"f64": 8, "f32": 4, "mixed": 4, "mixed_bf16": 2}[case["prec"]]
    xb = 8 if case["prec"] == "f64" else 4
    if case["kind"] == "batched":
        g = torch.Generator()
        g.manual_seed(case["count"] * 1000003 + case["n_hi"])
        ns = torch.exp(math.log(case["n_lo"]) + torch.rand(case["count"], generator=g, dtype=torch.float64)
                       * math.log(case["n_hi"] / case["n_lo"])).long()
        avg = 4.0 + 60.0 * torch.rand(case["count"], generator=g, dtype=torch.float64)
        n, nz, k = int(ns.sum()), int((ns * avg).sum()), case["k"]
        return {"bytes": (4 + vb) * nz + 4 * (n + case["count"]) + 2 * xb * k * n, "flops": 2 * nz * k}
    n, nz = _shape(case)
    if case["kind"] == "spmv":
        return {"bytes": (4 + vb) * nz + 4 * (n + 1) + 2 * xb * n, "flops": 2 * nz}
    if case["kind"] == "grad":
        # forward: A, x, y; dx: A^T's columns and row pointers, the values
        # again with their permutation, g, dx; dvalues: the pattern, g, x, dv
        fwd = (4 + vb) * nz + 4 * (n + 1) + 2 * xb * n
        dx = (8 + vb) * nz + 4 * (n + 1) + 2 * xb * n
        dv = (4 + vb) * nz + 4 * (n + 1) + 2 * xb * n
        return {"bytes": fwd + dx + dv, "flops": 5 * nz}
    # CG: iterations from the condition number; per iteration the matrix, x,
    # r and p read and written, q written and read
    kappa = (8.0 + CG_SHIFT) / CG_SHIFT
    it = math.ceil(math.sqrt(kappa) / 2.0 * math.log(2.0 / (1e-8 if case["prec"] == "f64" else 1e-5)))
    return {"bytes": it * ((4 + vb) * nz + 4 * (n + 1) + 8 * xb * n), "flops": it * (2 * nz + 10 * n)}


# ------------------------------------------------------------------ exact


def _product(Rst, Col, Val, x):
    """A x in fp64; x may hold several columns."""
    row = _row_of(Rst)
    out = torch.zeros((Rst.numel() - 1,) + x.shape[1:], dtype=torch.float64, device=x.device)
    step = 1 << 26
    for a in range(0, Col.numel(), step):
        v = Val[a:a + step].double()
        p = x[Col[a:a + step].long()].double()
        out.index_add_(0, row[a:a + step], p * (v if x.dim() == 1 else v[:, None]))
    return out


def _dst_solve(b, side):
    """(L + CG_SHIFT) x = b for the Dirichlet Laplacian L by sine transforms."""
    def dst(a):  # along the last axis: the imaginary part of an odd extension's transform
        z = torch.zeros(a.shape[0], 2 * side + 2, dtype=torch.float64, device=a.device)
        z[:, 1:side + 1] = a
        z[:, side + 2:] = -a.flip(1)
        return torch.fft.rfft(z, dim=1).imag[:, 1:side + 1]

    i = torch.arange(1, side + 1, dtype=torch.float64, device=b.device)
    lam = 2.0 - 2.0 * torch.cos(math.pi * i / (side + 1))
    f = dst(dst(b.double().view(side, side)).T.contiguous()) / (lam[:, None] + lam[None, :] + CG_SHIFT)
    return (dst(dst(f).T.contiguous()) / (4.0 * (side + 1) ** 2)).reshape(-1)


def exact(case, seed):
    d = _inputs(case, seed)
    if case["kind"] == "spmv":
        return _product(d["Rst"], d["Col"], d["Val"], d["x"])
    if case["kind"] == "grad":
        row, col = _row_of(d["Rst"]), d["Col"].long()
        g, x, v = d["g"].double(), d["x"].double(), d["Val"].double()
        dx = torch.zeros_like(x).index_add_(0, col, g[row] * v)
        return {"y": _product(d["Rst"], d["Col"], d["Val"], d["x"]), "dvalues": g[row] * x[col], "dx": dx}
    if case["kind"] == "batched":
        k = case["k"]
        mat = torch.repeat_interleave(torch.arange(len(d["ns"])), torch.tensor(d["ns"])).cuda()
        base = torch.tensor(d["start"][:-1]).cuda()[mat]
        col = d["Col"].long() + base[_row_of(d["Rst"])]
        x = d["x"] if k == 1 else d["x"].view(-1, k)
        return _product(d["Rst"], col, d["Val"], x).reshape(-1)
    return {"x": _dst_solve(d["x"], case["n"]), "iterations": None}
