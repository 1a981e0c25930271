"""A solve whose basis outgrows the resident kernel (10240 columns): the
intervals up to there are resident, the rest runs on the kernel chain from the
state that the resident kernel left, and the solve is the one that the chain
makes alone (use_graphs = 0)."""
import pytest
import torch

from test_gpu_parity import csr_tensor

pytestmark = pytest.mark.gpu


def test_the_chain_goes_on_where_the_resident_kernel_ends():
    """22000 launches tell the paths apart.  Column scales over three decades:
    the condition is below 1e4, so that x is fixed to 4e4 times the backward
    error that both solves report."""
    import amfls_solver_gb300 as amfls
    from amfls_solver_gb300 import _native, binding, problems

    p = problems.scaled_uniform_csr(21200, 10600, per_row=6, decades=3.0, noise=1e-10, seed=1)
    op, b = amfls.DeviceOperator(csr_tensor(p)), torch.from_numpy(p.b).cuda()
    runs = []
    for graphs in (1, 0):
        o = _native.default_options()
        o.tolerance, o.maximum_depth, o.use_graphs = 1e-15, 10400, graphs
        native = []
        r = binding._decode(binding._solve_raw("amfls", op, b, o, native))
        runs.append((r, native[0].kernel_launches))
    (r, few), (chain, many) = runs
    # ten kernels or more a level on the chain: 8192 levels of the first solve have none
    assert 10 * (10400 - 8192) < few < many - 10 * 8192
    assert (r.status, r.stop_reason, r.iterations) == (
        chain.status, chain.stop_reason, chain.iterations) == (1, 3, 10400)
    bound = r.backward_error_upper_bound
    assert abs(bound - chain.backward_error_upper_bound) <= 1e-3 * bound
    x, y = r.solution, chain.solution
    assert torch.linalg.norm(x - y) <= 4e4 * bound * torch.linalg.norm(y)
