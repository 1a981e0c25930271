"""Projected solves of width-one levels (lambda = 0) in which rhobar = q^(1/2) falls
below 1e-154 within one interval: 1 / q leaves FP64's range there, rhobar does
not.  A is itself lower bidiagonal and b = e_1, so that T = A without rounding
and y_j = (-1)^j prod(beta / alpha) solves T y = e_1."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def bidiagonal(beta):
    """alpha = 1 on the diagonal, beta below it."""
    n = len(beta) + 1
    off = np.concatenate([[0, 1], 1 + 2 * np.arange(1, n)]).astype(np.int64)
    idx, val = [0], [1.0]
    for i in range(1, n):
        idx += [i - 1, i]
        val += [beta[i - 1], 1.0]
    return torch.sparse_csr_tensor(torch.from_numpy(off), torch.tensor(idx),
                                   torch.tensor(val, dtype=torch.float64), size=(n, n)).cuda()


@pytest.mark.parametrize("steep,ratio", [(10, 1e6), (24, 1e6), (30, 1e6), (36, 1e6), (45, 1e4)])
def test_square_systems(steep, ratio):
    """phibar falls by half in each of the first 256 columns, so that y stays
    small enough for a finite ||x||^2; 24 columns of ratio 1e6 stay within 1 / q's
    range, the others do not.  The levels end at the basis limit."""
    import amfls_solver_gb300 as amfls

    beta = np.concatenate([np.full(256, 0.5), np.full(steep, ratio)])
    a = bidiagonal(beta)
    b = torch.zeros(a.shape[0], dtype=torch.float64, device="cuda")
    b[0] = 1.0
    r = amfls.run_amfls(a, b, tolerance=1e-300)
    assert (r.status, r.stop_reason) == (2, 5)
    x = r.solution.cpu().numpy()
    y = np.cumprod(np.concatenate([[1.0], -beta]))[:r.depth]
    assert np.all(np.isfinite(x))
    # T y = e_1 is solved by products of positive terms alone: n roundings each
    if r.depth == a.shape[1]:
        assert np.all(np.abs(x - y) <= 1e-12 * np.abs(y))
