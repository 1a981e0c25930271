"""Performance cases of the AMFLS solver: what is measured, and on which inputs.

A case is one call a user's program makes, on seeded synthetic inputs of the
families the benchmark and the tests use: a solve to tolerance (AMFLS on CSR
operators, its mixed-precision form, a batch of small problems, fixed-width
RBGK, scalar LSQR / LSMR) or a pair of operator products (A X and A^T Y).

CSR matrices: `per_row` nonzeros per row at uniform columns, or `per_row` 0 for
power-law row lengths (tail exponent 1.5, mean 20, at most 2000); N(0,1) values
with column j scaled by 10^(-decades j / n); b = A x_true + noise.  Dense
matrices: i.i.d. N(0,1) with the same column scaling.

The solve cases are conditioned, and solved far enough, that x is settled to
about 1e-10 whatever the order of its sums (an unregularised problem of
condition 1e6 leaves x open by 1e-8 to 1e-2).
"""
import math

import numpy as np
import torch

import amfls_solver_gb300 as amfls


# ------------------------------------------------------------------ inputs

def _generator(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + 7919 * salt + 11) % (1 << 62))
    return g


def _csr(rows, cols, per_row, decades, g):
    """Row offsets, column indices (sorted, distinct within a row), values."""
    if per_row:
        lengths = torch.full((rows,), min(per_row, cols), dtype=torch.int64, device="cuda")
    else:
        u = 1.0 - torch.rand(rows, dtype=torch.float64, device="cuda", generator=g)
        lengths = torch.ceil(0.04688 * u ** -2.0).clamp_(1, min(2000, cols)).to(torch.int64)
    row = torch.repeat_interleave(torch.arange(rows, device="cuda"), lengths)
    col = torch.randint(0, cols, (row.numel(),), device="cuda", generator=g)
    key = torch.unique(row * cols + col)  # sorted; a repeated column of a row is dropped
    row = torch.div(key, cols, rounding_mode="floor")
    col = key - row * cols
    offsets = torch.zeros(rows + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(torch.bincount(row, minlength=rows), 0, out=offsets[1:])
    values = torch.randn(col.numel(), dtype=torch.float64, device="cuda", generator=g)
    values *= 10.0 ** (-decades * col.to(torch.float64) / cols)
    return offsets, row, col, values


def _matvec(row, col, values, rows, x):
    return torch.zeros(rows, dtype=torch.float64, device="cuda").index_add_(0, row, values * x[col])


def _system(case, seed, salt=0):
    """The matrix tensor and b of a solve case."""
    rows, cols = case["rows"], case["cols"]
    g = _generator(seed, salt)
    x_true = torch.randn(cols, dtype=torch.float64, device="cuda", generator=g)
    if case["matrix"] == "csr":
        offsets, row, col, values = _csr(rows, cols, case["per_row"], case["decades"], g)
        a = torch.sparse_csr_tensor(offsets, col, values, size=(rows, cols))
        # the same sums on every run: a segment sum, not atomic additions
        b = torch.segment_reduce(values * x_true[col], "sum", offsets=offsets, initial=0.0)
    else:
        a = _dense(case, g)
        b = a @ x_true
    b = b + case["noise"] * torch.randn(rows, dtype=torch.float64, device="cuda", generator=g)
    return a, b


def _dense(case, g):
    rows, cols = case["rows"], case["cols"]
    a = torch.randn(rows, cols, dtype=torch.float64, device="cuda", generator=g)
    a *= 10.0 ** (-case["decades"] * torch.arange(cols, dtype=torch.float64, device="cuda")
                  / max(1, cols - 1))
    # column-major: the transpose of a contiguous tensor
    return a.t().contiguous().t() if case["matrix"] == "dense_columns" else a


def _batch_sizes(case):
    """The (rows, cols, per_row) of a batch's problems, log-uniform, fixed by the case."""
    rng = np.random.default_rng(case["count"] * 1000 + case["rows"])
    out = []
    for _ in range(case["count"]):
        m = int(np.exp(rng.uniform(np.log(case["rows"] / 10), np.log(case["rows"]))))
        n = int(np.exp(rng.uniform(np.log(case["cols"] / 10), np.log(case["cols"]))))
        out.append((m, max(1, min(n, m // 2)), int(rng.integers(5, 41))))
    return out


# ------------------------------------------------------------------- cases

def listed():
    return [
        # smallest solve of the batched workload's family, straight from tensors: operator
        # construction, launches and latency
        dict(name="amfls_2000x500", call="run_amfls", matrix="csr", rows=2000, cols=500,
             per_row=10, decades=2.0, noise=1e-6, reg=1e-2, tol=1e-10),
        # the headline benchmark's shape, least squares, on a kept operator
        dict(name="amfls_20000x5000", call="amfls", matrix="csr", rows=20000, cols=5000,
             per_row=10, decades=2.0, noise=1e-12, reg=0.0, tol=1e-11),
        # the tall ridge problem of the parity fixtures, to its 1e-10
        dict(name="amfls_60000x15000_ridge", call="amfls", matrix="csr", rows=60000, cols=15000,
             per_row=10, decades=6.0, noise=1e-6, reg=1e-3, tol=1e-10),
        # the chosen mixed form at a tenth of the 2M x 500k power-law workload: FP64 products,
        # FP16 copy of the basis, restart cycles
        dict(name="mixed_200000x50000", call="mixed", matrix="csr", rows=200000, cols=50000,
             per_row=0, decades=8.0, noise=1e-6, reg=1e-2, tol=1e-10, values="fp64",
             basis="fp16", cycle=500),
        # independent problems of uneven size, solved together
        dict(name="batch_16", call="batch", matrix="csr", rows=20000, cols=4000, count=16,
             workers=16, decades=3.0, noise=1e-8, reg=1e-2, tol=1e-10),
        # block levels (width 8) on a CSR operator
        dict(name="rbgk_5000x1200_w8", call="rbgk", matrix="csr", rows=5000, cols=1200,
             per_row=8, decades=2.0, noise=1e-6, reg=1e-2, tol=1e-10, width=7),
        # block levels (width 4) on the dense study's tall shape, row-major as torch gives it
        dict(name="rbgk_dense_16384x512_w4", call="rbgk", matrix="dense_rows", rows=16384,
             cols=512, decades=2.0, noise=1e-6, reg=1e-2, tol=1e-10, width=3),
        # the scalar baseline solvers on the headline shape
        dict(name="lsmr_20000x5000", call="lsmr", matrix="csr", rows=20000, cols=5000,
             per_row=10, decades=2.0, noise=1e-8, reg=1e-2, tol=1e-11),
        # single-column products of the large power-law matrix, both directions
        dict(name="spmv_1000000x250000", call="apply", matrix="csr", rows=1000000, cols=250000,
             per_row=0, decades=8.0, block=1, values="fp64"),
        # eight-column products: block levels, validation of several candidates
        dict(name="spmm_200000x50000_s8", call="apply", matrix="csr", rows=200000, cols=50000,
             per_row=0, decades=8.0, block=8, values="fp64"),
        # the dense benchmark's products, FP64, row-major
        dict(name="dense_100000x2000_s1", call="apply", matrix="dense_rows", rows=100000,
             cols=2000, decades=6.0, block=1, values="fp64"),
        # the reduced copy the mixed form multiplies by, column-major
        dict(name="dense_fp32_100000x2000_s1", call="apply", matrix="dense_columns", rows=100000,
             cols=2000, decades=6.0, block=1, values="fp32"),
    ]


def draw(rng):
    """One more case of the listed ones' ranges."""
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["amfls", "amfls", "amfls", "mixed", "batch", "rbgk", "rbgk_dense",
                       "baseline", "spmv", "spmm", "dense"])
    if kind == "amfls":
        rows = log(2000, 60000)
        reg = rng.choice([0.0, 1e-3, 1e-2])
        return dict(call=rng.choice(["run_amfls", "amfls"]), matrix="csr", rows=rows,
                    cols=log(500, max(501, rows // 4)), per_row=rng.choice([0, rng.randint(5, 40)]),
                    decades=round(rng.uniform(0.5, 2.0 if reg == 0.0 else 6.0), 2),
                    noise=1e-12 if reg == 0.0 else 1e-6, reg=reg,
                    tol=1e-11 if reg == 0.0 else 1e-10)
    if kind == "mixed":
        rows = log(20000, 200000)
        return dict(call="mixed", matrix="csr", rows=rows, cols=rows // rng.randint(4, 6),
                    per_row=0, decades=round(rng.uniform(3.0, 8.0), 2), noise=1e-6, reg=1e-2,
                    tol=1e-10, values="fp64", basis=rng.choice(["fp16", "fp32"]),
                    cycle=rng.randint(300, 600))
    if kind == "batch":
        rows = log(5000, 20000)
        return dict(call="batch", matrix="csr", rows=rows, cols=rows // 5,
                    count=rng.randint(4, 16), workers=rng.choice([4, 8, 16]),
                    decades=round(rng.uniform(1.0, 3.0), 2), noise=1e-8,
                    reg=rng.choice([1e-3, 1e-2]), tol=1e-10)
    if kind == "rbgk":
        rows = log(2000, 20000)
        return dict(call="rbgk", matrix="csr", rows=rows, cols=log(400, max(401, rows // 8)),
                    per_row=rng.randint(5, 20), decades=round(rng.uniform(1.0, 2.5), 2),
                    noise=1e-6, reg=rng.choice([1e-3, 1e-2]), tol=1e-10,
                    width=rng.randint(1, 15))
    if kind == "rbgk_dense":
        return dict(call="rbgk", matrix=rng.choice(["dense_rows", "dense_columns"]),
                    rows=log(1000, 16384), cols=log(100, 512),
                    decades=round(rng.uniform(1.0, 2.5), 2), noise=1e-6,
                    reg=rng.choice([1e-3, 1e-2]), tol=1e-10, width=rng.choice([0, 1, 3, 7]))
    if kind == "baseline":
        rows = log(2000, 60000)
        return dict(call=rng.choice(["lsqr", "lsmr"]), matrix="csr", rows=rows,
                    cols=log(500, max(501, rows // 4)), per_row=rng.randint(5, 40),
                    decades=round(rng.uniform(0.5, 2.0), 2), noise=1e-8,
                    reg=rng.choice([1e-3, 1e-2]), tol=1e-11)
    if kind in ("spmv", "spmm"):
        rows = log(2000, 1000000 if kind == "spmv" else 200000)
        return dict(call="apply", matrix="csr", rows=rows, cols=max(500, rows // rng.randint(2, 8)),
                    per_row=rng.choice([0, rng.randint(5, 40)]) if rows < 400000 else 0,
                    decades=round(rng.uniform(1.0, 8.0), 2),
                    block=1 if kind == "spmv" else rng.randint(2, 11),
                    values=rng.choice(["fp64", "fp64", "fp32", "bf16"]))
    return dict(call="apply", matrix=rng.choice(["dense_rows", "dense_columns"]),
                rows=log(1000, 100000), cols=log(100, 2000),
                decades=round(rng.uniform(0.0, 6.0), 2), block=rng.choice([1, 1, 2, 4]),
                values=rng.choice(["fp64", "fp64", "fp32", "bf16"]))


# --------------------------------------------------------------- interface

def prepare(case, seed):
    if case["call"] == "apply":
        g = _generator(seed)
        if case["matrix"] == "csr":
            offsets, _, col, values = _csr(case["rows"], case["cols"], case["per_row"],
                                           case["decades"], g)
            a = torch.sparse_csr_tensor(offsets, col, values, size=(case["rows"], case["cols"]))
        else:
            a = _dense(case, g)
        s = case["block"]
        x = torch.randn(case["cols"], s, dtype=torch.float64, device="cuda", generator=g)
        y = torch.randn(case["rows"], s, dtype=torch.float64, device="cuda", generator=g)
        if s == 1:
            x, y = x.reshape(-1), y.reshape(-1)
        op = amfls.DeviceOperator(a)
        if case["values"] != "fp64":
            op = op.reduced(case["values"])
        return dict(case=case, op=op, x=x, y=y)
    if case["call"] == "batch":
        problems = []
        for i, (m, n, per_row) in enumerate(_batch_sizes(case)):
            a, b = _system(dict(case, rows=m, cols=n, per_row=per_row), seed, i + 1)
            problems.append((amfls.DeviceOperator(a), b))
        return dict(case=case, problems=problems)
    a, b = _system(case, seed)
    keep = case["call"] in ("amfls", "mixed")
    return dict(case=case, a=amfls.DeviceOperator(a) if keep else a, b=b)


def _answer(r):
    # the depth stays out: a solve stops at a checkpoint predicted by the ceiling of a ratio of
    # logarithms of certificates, which another order of the same sums can move by a level; so
    # do the norms of a residual that tends to zero
    return dict(solution=r.solution, status=r.status, stop_reason=r.stop_reason,
                solution_norm=r.solution_norm)


def run(state):
    case = state["case"]
    call = case["call"]
    if call == "apply":
        return dict(ax=state["op"].apply(state["x"]),
                    aty=state["op"].apply(state["y"], transpose=True))
    if call == "batch":
        results, _, _ = amfls.run_amfls_batch(state["problems"], workers=case["workers"],
                                              regularization=case["reg"], tolerance=case["tol"])
        return [dict(solution=r.solution, status=r.status) for r in results]
    opts = dict(regularization=case["reg"], tolerance=case["tol"])
    a, b = state["a"], state["b"]
    if call == "run_amfls":
        r = amfls.run_amfls(a, b, **opts)
    elif call == "amfls":
        r = amfls.solve_amfls(a, b, **opts)
    elif call == "mixed":
        r = amfls.run_amfls_mixed(a, b, values=case["values"], reduced_basis=case["basis"],
                                  inner_tolerance=1e-14, maximum_refinements=40,
                                  maximum_depth=case["cycle"], **opts)
    elif call == "rbgk":
        r = amfls.run_fixed_rbgk(a, b, auxiliary_width=case["width"],
                                 maximum_depth=min(case["rows"], case["cols"]), **opts)
    elif call == "lsqr":
        r = amfls.run_lsqr(a, b, **opts)
    else:
        r = amfls.run_lsmr(a, b, **opts)
    return _answer(r)


def work(case):
    """Each input read once and each output written once; for a solve, the
    operations of one product pair alone (how many levels it takes is the
    problem's matter)."""
    def system(rows, cols, per_row):
        if case["matrix"] != "csr":
            return 8.0 * rows * cols, 4.0 * rows * cols
        nnz = rows * float(per_row or 20)
        return 12.0 * nnz + 4.0 * rows, 4.0 * nnz

    if case["call"] == "batch":
        parts = [(system(m, n, p), 8.0 * (m + n)) for m, n, p in _batch_sizes(case)]
        return {"bytes": sum(a[0] + v for a, v in parts), "flops": sum(a[1] for a, _ in parts)}
    rows, cols = case["rows"], case["cols"]
    nbytes, flops = system(rows, cols, case.get("per_row"))
    if case["call"] != "apply":
        return {"bytes": nbytes + 8.0 * (rows + cols), "flops": flops}
    width = {"fp64": 8.0, "fp32": 4.0, "bf16": 2.0}[case["values"]]
    if case["matrix"] == "csr":
        nbytes = nbytes / 12.0 * (4.0 + width)
    else:
        nbytes = nbytes / 8.0 * width
    s = case["block"]
    return {"bytes": 2.0 * nbytes + 16.0 * s * (rows + cols), "flops": flops * s}


# ------------------------------------------------------------ 64-bit values

def _transposed(row, col, values, rows, cols):
    order = torch.argsort(col * rows + row)
    offsets = torch.zeros(cols + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(torch.bincount(col, minlength=cols), 0, out=offsets[1:])
    return torch.sparse_csr_tensor(offsets, row[order], values[order], size=(cols, rows))


def _ridge_solution(a, b, reg):
    """argmin ||A x - b||^2 + reg ||x||^2 in 64 bits: corrections by a factor of
    the column-scaled normal equations (small) or by conjugate gradients on
    them, with residuals of the original system until they no longer shrink."""
    rows, cols = a.shape
    if a.layout == torch.sparse_csr:
        row = torch.repeat_interleave(torch.arange(rows, device="cuda"),
                                      a.crow_indices().diff())
        at = _transposed(row, a.col_indices(), a.values(), rows, cols)
        square = torch.zeros(cols, dtype=torch.float64, device="cuda").index_add_(
            0, a.col_indices(), a.values() ** 2)
    else:
        at = a.t()
        square = (a * a).sum(0)
    scale = 1.0 / torch.sqrt(square + reg).clamp_min(1e-150)
    factor = None
    if cols <= 6000:
        dense = (a.to_dense() if a.layout == torch.sparse_csr else a) * scale
        h = dense.t() @ dense
        h += torch.diag(reg * scale * scale)
        del dense
        factor = torch.linalg.cholesky(h)
    x = torch.zeros(cols, dtype=torch.float64, device="cuda")
    last = math.inf
    for _ in range(12):
        g = (at @ (b - a @ x) - reg * x) * scale
        if factor is not None:
            d = torch.cholesky_solve(g[:, None], factor)[:, 0]
        else:
            d = _conjugate_gradients(a, at, scale, reg, g)
        d = d * scale
        size = float(d.norm() / (x + d).norm())
        if size >= 0.5 * last:
            break
        x, last = x + d, size
    return x


def _conjugate_gradients(a, at, scale, reg, g):
    x, r, p = torch.zeros_like(g), g.clone(), g.clone()
    rr = torch.dot(r, r)
    stop = 1e-10 * float(rr)
    for i in range(20000):
        q = scale * (at @ (a @ (scale * p))) + reg * scale * scale * p
        alpha = rr / torch.dot(p, q)
        x, r = x + alpha * p, r - alpha * q
        new = torch.dot(r, r)
        if i % 50 == 49 and not float(new) > stop:
            break
        p, rr = r + (new / rr) * p, new
    return x


def exact(case, seed):
    if case["call"] == "apply":
        g = _generator(seed)
        rows, cols, s = case["rows"], case["cols"], case["block"]
        if case["matrix"] == "csr":
            _, row, col, values = _csr(rows, cols, case["per_row"], case["decades"], g)
        else:
            a = _dense(case, g)
        x = torch.randn(cols, s, dtype=torch.float64, device="cuda", generator=g)
        y = torch.randn(rows, s, dtype=torch.float64, device="cuda", generator=g)
        if case["matrix"] == "csr":
            ax = torch.stack([_matvec(row, col, values, rows, x[:, c]) for c in range(s)], 1)
            aty = torch.stack([_matvec(col, row, values, cols, y[:, c]) for c in range(s)], 1)
        else:
            ax, aty = a @ x, a.t() @ y
        if s == 1:
            ax, aty = ax.reshape(-1), aty.reshape(-1)
        return dict(ax=ax, aty=aty)
    if case["call"] == "batch":
        out = []
        for i, (m, n, per_row) in enumerate(_batch_sizes(case)):
            a, b = _system(dict(case, rows=m, cols=n, per_row=per_row), seed, i + 1)
            out.append(dict(solution=_ridge_solution(a, b, case["reg"])))
        return out
    a, b = _system(case, seed)
    x = _ridge_solution(a, b, case["reg"])
    return dict(solution=x, solution_norm=float(x.norm()))
