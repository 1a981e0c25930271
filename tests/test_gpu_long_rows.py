"""Solves on CSR matrices with one dense column or row.  In the resident kernels a
row is one warp's and every other block waits for it, so beyond the measured
limits (18000 nonzeros more than an even share for AMFLS levels, 42000 for LSQR
and LSMR) the general paths, whose tiles slice long rows, take the solve.
Which path ran shows in the kernels launched: the general ones launch more than
ten per level.  On either side of the limits the outcome is the oracle's."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import amfls_oracle as orc
from oracle import baselines as orc_baselines
from test_gpu_parity import check_solution, csr_tensor

pytestmark = pytest.mark.gpu

ROWS, COLS, REG, TOL = 60000, 200, 1e-2, 1e-9


def with_dense_column(length):
    """Three nonzeros a row at distinct columns 1 .., and `length` in column 0."""
    from amfls_solver_gb300 import problems

    rng = np.random.default_rng(length)
    col = 1 + (rng.integers(0, COLS - 1, ROWS)[:, None] + np.array([0, 31, 77])) % (COLS - 1)
    has = np.zeros(ROWS, dtype=bool)
    has[rng.permutation(ROWS)[:length]] = True
    rows = [np.concatenate([[0], np.sort(c)]) if h else np.sort(c) for c, h in zip(col, has)]
    off = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    idx = np.concatenate(rows).astype(np.int64)
    val = rng.standard_normal(idx.size) * 10.0 ** (-3.0 * idx / COLS)
    p = problems.CsrProblem(ROWS, COLS, off, idx, val, np.zeros(ROWS))
    p.b = p.matvec(rng.standard_normal(COLS)) + 1e-3 * rng.standard_normal(ROWS)
    return p


def solve(method, op, b):
    from amfls_solver_gb300 import _native, binding

    lib = _native.load()
    o = _native.default_options() if method == "amfls" else _native.BaselineOptions()
    if method != "amfls":
        lib.amfls_gpu_default_baseline_options(ctypes.byref(o))
        o.maximum_iterations = 4000
    o.regularization, o.tolerance = REG, TOL
    native = []
    r = binding._decode(binding._solve_raw(method, op, b, o, native))
    return r, native[0].kernel_launches


@pytest.mark.parametrize("method,limit", [("amfls", 18000), ("lsqr", 42000), ("lsmr", 42000)])
@pytest.mark.parametrize("length", [10000, 30000, 60000])
def test_dense_column(method, limit, length):
    import amfls_solver_gb300 as amfls

    p = with_dense_column(length)
    r, launches = solve(method, amfls.DeviceOperator(csr_tensor(p)), torch.from_numpy(p.b).cuda())
    assert (launches > 10 * r.depth) == (length > limit)
    o = {"amfls": orc.solve_amfls, "lsqr": orc_baselines.solve_lsqr,
         "lsmr": orc_baselines.solve_lsmr}[method](
             p, regularization=REG, tolerance=TOL,
             **({} if method == "amfls" else dict(maximum_iterations=4000)))
    assert (r.status, r.stop_reason) == (o["status"], o["stop_reason"])
    check_solution(p, r.solution.cpu().numpy(), np.asarray(o["solution"]), REG, TOL,
                   r.status == 0)


def test_dense_row():
    """The same rule for A's rows."""
    import amfls_solver_gb300 as amfls

    rows, cols = 300, 30000
    rng = np.random.default_rng(1)
    idx = [np.sort(rng.choice(cols, 40, replace=False)) for _ in range(rows)]
    for long_row, resident in ((10000, True), (25000, False)):
        idx[7] = np.sort(rng.choice(cols, long_row, replace=False))
        off = np.concatenate([[0], np.cumsum([len(r) for r in idx])])
        a = torch.sparse_csr_tensor(torch.from_numpy(off), torch.from_numpy(np.concatenate(idx)),
                                    torch.from_numpy(rng.standard_normal(off[-1])),
                                    size=(rows, cols)).cuda()
        b = torch.from_numpy(rng.standard_normal(rows)).cuda()
        r, launches = solve("amfls", amfls.DeviceOperator(a), b)
        assert r.status == 0
        assert (launches > 10 * r.depth) == (not resident)
        x = r.solution
        y = a.to(torch.float64) @ x
        # the certificate bounds the gradient: ||A^T (A x - b) + reg x|| against both terms
        g = a.to_dense().t() @ (y - b) + REG * x
        assert torch.linalg.norm(g) <= 1e-6 * torch.linalg.norm(a.to_dense().t() @ b)
