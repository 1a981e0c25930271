"""GPU tests of solves whose magnitudes leave the range of the short cuts: plain
sums of squares in the validation (largest magnitudes within 2^-300 .. 2^300)
and the ratio recurrence of the projected solve (entries of T within 1e-15 ..
1e15).  A power of two scales A, b and lambda exactly, so the scaled problem is
the same problem: status, stop reason and depth must be those of the unscaled
solve, and x, scaled back, must agree as far as both certificates say
(2 tol in the energy norm for lambda > 0, 4 cond tol for lambda = 0)."""
import numpy as np
import pytest
import torch

from test_gpu_parity import csr_tensor
from test_gpu_resident import ragged_csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("reg", [0.0, 1e-2])
@pytest.mark.parametrize("a_exp,b_exp", [(0, -330), (0, 330), (60, 0), (-60, 0), (52, -320)])
def test_scaled_problem_is_the_same_problem(reg, a_exp, b_exp):
    import amfls_solver_gb300 as amfls

    p = ragged_csr(900, 260, [5, 8, 20], seed=11)
    if reg == 0.0:  # a consistent system, certified by its residual
        p.b = p.matvec(np.random.default_rng(2).standard_normal(p.cols))
    tol = 1e-9
    b = torch.from_numpy(p.b).cuda()
    base = amfls.run_amfls(csr_tensor(p), b, regularization=reg, tolerance=tol)
    values = p.values
    p.values = np.ldexp(values, a_exp)
    scaled = amfls.run_amfls(csr_tensor(p), torch.ldexp(b, torch.tensor(b_exp)),
                             regularization=float(np.ldexp(reg, 2 * a_exp)), tolerance=tol)
    p.values = values
    assert base.status == 0
    assert (scaled.status, scaled.stop_reason, scaled.depth) == (
        base.status, base.stop_reason, base.depth)
    x = base.solution.cpu().numpy()
    y = np.ldexp(scaled.solution.cpu().numpy(), a_exp - b_exp)
    a = p.to_dense()
    if reg > 0.0:
        h = lambda v: np.sqrt(np.linalg.norm(a @ v) ** 2 + reg * np.linalg.norm(v) ** 2)
        assert h(x - y) <= 2 * tol * h(x)
    else:
        s = np.linalg.svd(a, compute_uv=False)
        assert np.linalg.norm(x - y) <= 4 * s[0] / s[-1] * tol * np.linalg.norm(x)
