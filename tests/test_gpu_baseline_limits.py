"""LSQR and LSMR with iteration limits whose half-steps pass 2^31: the limit is
never reached, so the solve is the one without it."""
import pytest
import torch

from test_gpu_parity import csr_tensor
from test_gpu_resident import ragged_csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", ["run_lsqr", "run_lsmr"])
@pytest.mark.parametrize("limit", [2 ** 30 - 1, 2 ** 30, 2 ** 31 - 1])
def test_limits_beyond_half_the_int_range(method, limit):
    import amfls_solver_gb300 as amfls

    p = ragged_csr(700, 152, [8, 9, 16, 17], seed=5)
    a, b = csr_tensor(p), torch.from_numpy(p.b).cuda()
    opts = dict(regularization=1e-2, tolerance=1e-8)
    want = getattr(amfls, method)(a, b, maximum_iterations=2000, **opts)
    got = getattr(amfls, method)(a, b, maximum_iterations=limit, **opts)
    assert want.status == 0 and want.depth > 1
    assert (got.status, got.stop_reason, got.depth) == (want.status, want.stop_reason, want.depth)
    assert torch.equal(got.solution, want.solution)
