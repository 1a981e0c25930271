"""GPU tests of the block levels that run without host decisions (2 to 16
columns) where they can go wrong: every padding of the width and its edges, the
widths on either side of the range, bases that end inside a panel, blocks wider
than what is left of the space, rank-deficient matrices (where the
rank-revealing path has to take over), wide and dense problems.  Status, stop
reason, depth, basis rank and product counts must be the oracle's, and x must
pass the checks of the parity tests."""
import numpy as np
import pytest
import torch

from oracle import amfls_oracle as orc
from test_gpu_parity import _matrix_tensor, check_solution, csr_tensor
from test_gpu_resident import ragged_csr

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def amfls():
    import amfls_solver_gb300 as m

    m.load_library()
    return m


def solve_both(amfls, p, matrix, width, reg, tol=1e-8, depth=200, counts=True):
    opts = dict(auxiliary_width=width, regularization=reg, tolerance=tol, seed=5,
                maximum_depth=depth)
    r = amfls.run_fixed_rbgk(matrix, torch.from_numpy(p.b).cuda(), **opts)
    o = orc.solve_fixed_rbgk(p, **opts)
    assert (r.status, r.stop_reason) == (o["status"], o["stop_reason"])
    if counts:
        assert (r.depth, r.basis_rank) == (o["counters"][9], o["counters"][11])
        assert (r.search_a_columns, r.search_at_columns) == (o["counters"][4], o["counters"][5])
    check_solution(p, r.solution.cpu().numpy(), o["solution"], reg, tol, r.status == 0)
    return r


@pytest.mark.parametrize("reg", [0.0, 1e-2])
@pytest.mark.parametrize("width", [1, 2, 3, 4, 5, 7, 8, 9, 14, 15, 16, 17])
def test_widths_match_oracle(amfls, width, reg):
    p = ragged_csr(900, 305, [5, 33, 64, 65], seed=width)
    solve_both(amfls, p, csr_tensor(p), width, reg)


@pytest.mark.parametrize("rows,cols,lengths", [
    (40, 3, [2]), (50, 17, [0, 3, 5]), (90, 33, [4]), (60, 200, [12]), (700, 64, [8, 9, 17])])
@pytest.mark.parametrize("width", [2, 7, 15])
def test_small_spaces_match_oracle(amfls, rows, cols, lengths, width):
    p = ragged_csr(rows, cols, lengths, seed=rows)
    solve_both(amfls, p, csr_tensor(p), width, 1e-2)


@pytest.mark.parametrize("width", [3, 8])
def test_repeated_columns_match_oracle(amfls, width):
    """Each column twice: the Krylov space has half the dimensions, and the last
    block loses rank (how much rounding it keeps is not determined)."""
    from amfls_solver_gb300 import problems

    q = ragged_csr(300, 40, [6, 9], seed=7)
    a = q.to_dense()
    p = problems.DenseProblem(np.concatenate([a, a], axis=1), q.b)
    solve_both(amfls, p, _matrix_tensor(p), width, 1e-2, counts=False)


@pytest.mark.parametrize("column_major", [False, True])
@pytest.mark.parametrize("width", [4, 5, 13])
def test_dense_widths_match_oracle(amfls, width, column_major):
    from amfls_solver_gb300 import problems

    p = problems.scaled_dense(2000, 120, decades=3.0, seed=7, column_major=column_major)
    solve_both(amfls, p, _matrix_tensor(p), width, 1e-4)
