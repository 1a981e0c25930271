"""GPU tests of the dense products at the edges of their split: outputs per
warp, chunks and their sums over both kinds of reduction, one to nine columns,
both layouts and directions, against numpy; and of solves whose certificate
needs the double-double products of long and short dimensions."""
import numpy as np
import pytest
import torch

from oracle import amfls_oracle as orc
from test_gpu_parity import _matrix_tensor, check_solution

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def amfls():
    import amfls_solver_gb300 as m

    m.load_library()
    return m


@pytest.mark.parametrize("column_major", [False, True])
@pytest.mark.parametrize("rows,cols", [
    (1, 1), (3, 5), (31, 33), (257, 9), (9, 511), (513, 512), (1025, 7), (16391, 13),
    (5, 20011), (2431, 1025)])
def test_products_match_numpy(amfls, rows, cols, column_major):
    """|y - y_numpy| within both sides' rounding: each sums n products with a
    relative error of at most n u, so 2 (n + 1) u |A| |x| bounds the difference."""
    rng = np.random.default_rng(rows + cols)
    a = rng.standard_normal((rows, cols))
    t = torch.from_numpy(a).cuda()
    op = amfls.DeviceOperator(t.t().contiguous().t() if column_major else t)
    u = 2.0 ** -53
    for s in range(1, 10):
        for transpose, mat in ((False, a), (True, a.T)):
            x = rng.standard_normal((mat.shape[1], s))
            y = op.apply(torch.from_numpy(x).cuda(), transpose=transpose).cpu().numpy()
            bound = 2 * (mat.shape[1] + 1) * u * (np.abs(mat) @ np.abs(x))
            assert y.shape == (mat.shape[0], s)
            assert np.all(np.abs(y - mat @ x) <= bound)


@pytest.mark.parametrize("column_major", [False, True])
@pytest.mark.parametrize("rows,cols", [(20011, 33), (700, 300), (64, 1500)])
def test_tight_certificates_match_oracle(amfls, rows, cols, column_major):
    from amfls_solver_gb300 import problems

    p = problems.scaled_dense(rows, cols, decades=1.0, seed=3, column_major=column_major)
    opts = dict(auxiliary_width=2, regularization=0.0, tolerance=1e-13, seed=5, maximum_depth=400)
    r = amfls.run_fixed_rbgk(_matrix_tensor(p), torch.from_numpy(p.b).cuda(), **opts)
    o = orc.solve_fixed_rbgk(p, **opts)
    assert r.status == o["status"] == 0
    check_solution(p, r.solution.cpu().numpy(), o["solution"], 0.0, 1e-13, True)
