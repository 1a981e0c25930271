"""Fixed-width block solves whose entries come near the ends of FP64's range.
A power of two scales A exactly, so x scales back exactly but for what the
squares lose below 2^-1022: sums of squares near 2^(2 e + 3) keep their bits
above 2^-1074.  The systems are consistent (condition below 10, rows of eight
entries), so x is known."""
import numpy as np
import pytest
import torch

from test_gpu_parity import csr_tensor
from test_gpu_resident import ragged_csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [1, 2, 5, 15])
@pytest.mark.parametrize("exponent", [-518, -516, -514, -505, -480, -300, 300, 480, 508])
def test_scaled_blocks_solve_the_same_problem(width, exponent):
    import amfls_solver_gb300 as amfls

    p = ragged_csr(300, 60, [8], seed=3)
    x = np.random.default_rng(1).standard_normal(p.cols)
    s = np.linalg.svd(p.to_dense(), compute_uv=False)
    cond = s[0] / s[-1]
    assert cond < 10
    b = p.matvec(x)
    p.values = np.ldexp(p.values, exponent)
    r = amfls.run_fixed_rbgk(csr_tensor(p), torch.from_numpy(b).cuda(), auxiliary_width=width,
                             maximum_depth=60, tolerance=1e-9)
    # a certified solve, or the full basis where the certificate's own squares underflow
    assert r.status in (0, 2)
    got = np.ldexp(r.solution.cpu().numpy(), exponent)
    bits = min(52, 2 * exponent + 3 + 1074)
    # 4 cond tol for the certificate; the squares' loss enters every norm, and the full
    # basis amplifies it by the condition of the normal equations
    bound = 4 * cond * 1e-9 + 100 * cond ** 2 * 2.0 ** -bits
    assert np.linalg.norm(got - x) <= bound * np.linalg.norm(x)
