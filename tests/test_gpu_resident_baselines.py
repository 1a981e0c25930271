"""GPU tests of the resident LSQR and LSMR iterations where they can go wrong:
fewer rows or columns than blocks, rows of every lane count, empty rows, wide
problems, limits that end on either half-step, breakdowns and magnitudes that
have to be handed back to the general path.  Status and stop reason must be
the oracle's, the depth too where a limit or a breakdown decides it, and x must
pass the checks of the parity tests."""
import numpy as np
import pytest
import torch

from oracle import baselines as orc
from test_gpu_parity import check_solution, csr_tensor
from test_gpu_resident import SIZES, ragged_csr

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def amfls():
    import amfls_solver_gb300 as m

    m.load_library()
    return m


def both(amfls, method, p, **opts):
    fn = dict(lsqr=amfls.run_lsqr, lsmr=amfls.run_lsmr)[method]
    ref = dict(lsqr=orc.solve_lsqr, lsmr=orc.solve_lsmr)[method]
    return fn(csr_tensor(p), torch.from_numpy(p.b).cuda(), **opts), ref(p, **opts)


@pytest.mark.parametrize("method", ["lsqr", "lsmr"])
@pytest.mark.parametrize("rows,cols,lengths", SIZES)
def test_solves_match_oracle(amfls, method, rows, cols, lengths):
    p = ragged_csr(rows, cols, lengths, seed=rows + cols)
    reg, tol = 1e-2, 1e-8
    r, o = both(amfls, method, p, regularization=reg, tolerance=tol, maximum_iterations=2000)
    assert (r.status, r.stop_reason) == (o["status"], o["stop_reason"])
    check_solution(p, r.solution.cpu().numpy(), np.asarray(o["solution"]), reg, tol,
                   r.status == 0)


@pytest.mark.parametrize("method", ["lsqr", "lsmr"])
@pytest.mark.parametrize("limit", [1, 2, 3, 17])
def test_limits_match_oracle(amfls, method, limit):
    """Before orthogonality is lost: x within 1e-8 of the oracle's, and the
    oracle's product counts."""
    p = ragged_csr(900, 305, [5, 33, 64, 65], seed=3)
    r, o = both(amfls, method, p, regularization=0.0, tolerance=1e-12, maximum_iterations=limit)
    c = o["counters"]
    assert (r.status, r.stop_reason, r.depth) == (o["status"], o["stop_reason"], c[9])
    assert (r.search_a_columns, r.search_at_columns) == (c[4], c[5])
    x, xr = r.solution.cpu().numpy(), np.asarray(o["solution"])
    assert np.linalg.norm(x - xr) <= 1e-8 * np.linalg.norm(xr)


@pytest.mark.parametrize("method", ["lsqr", "lsmr"])
@pytest.mark.parametrize("scale_a,scale_b", [(1.0, 1.0), (2.0 ** -400, 1.0), (2.0 ** 400, 1.0),
                                             (1.0, 2.0 ** -500), (2.0 ** 300, 2.0 ** -300)])
def test_breakdowns_and_magnitudes_match_oracle(amfls, method, scale_a, scale_b):
    """A multiple of the identity breaks down after one iteration; scaled
    problems leave the range of plain sums of squares."""
    from amfls_solver_gb300 import problems

    n = 70
    eye = problems.CsrProblem(n, n, np.arange(n + 1, dtype=np.int64), np.arange(n, dtype=np.int64),
                              np.full(n, scale_a), scale_b * np.arange(1.0, n + 1))
    q = ragged_csr(300, 40, [6, 9], seed=7)
    q.values = q.values * scale_a
    q.b = q.b * scale_b
    for p in (eye, q):
        r, o = both(amfls, method, p, regularization=0.0, tolerance=1e-9, maximum_iterations=300)
        assert (r.status, r.stop_reason) == (o["status"], o["stop_reason"])
        x, xr = r.solution.cpu().numpy(), np.asarray(o["solution"])
        if r.status == 0:
            assert np.max(np.abs(x / np.max(np.abs(xr)) - xr / np.max(np.abs(xr)))) <= 1e-6
