"""Levels on a reduced copy of the basis whose projection is redone in FP64.

The CPU model of the sweeps (oracle/reduced_sweeps.py) says how many levels of
two problems ask for it: a single deep solve, whose left basis loses
orthogonality (FP32 and FP16), and restart cycles with the FP16 copy that are
long for their problem.  On the GPU every block of the resident kernel must come
to the same decisions from the same sums: the levels that fell back are counted,
repeats give the same bits, and the restarted solve meets its certificate and
the oracle's x."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

from amfls_solver_gb300 import problems
from oracle import amfls_oracle as orc
from oracle import reduced_sweeps as rs

DEEP = dict(m=2000, n=320, per_row=10, decades=5.0, noise=1e-8, seed=3)
CYCLES = dict(m=2000, n=320, per_row=9, decades=2.0, noise=1e-6, seed=2000)
REG, CYCLE = 1e-3, 150


def csr_matrix(p):
    return sp.csr_matrix((p.values, p.column_indices, p.row_offsets), shape=(p.rows, p.cols))


def test_the_model_falls_back_in_a_deep_solve():
    p = problems.scaled_uniform_csr(**DEEP)
    for storage in ("fp32", "fp16"):
        gk = rs.GolubKahan(csr_matrix(p), 300, storage)
        gk.solve(p.b, 300)
        assert gk.reduced_passes == 299 and gk.fallbacks > 100


def test_the_model_falls_back_in_long_fp16_cycles():
    p = problems.scaled_uniform_csr(**CYCLES)
    m = sp.vstack([csr_matrix(p), np.sqrt(REG) * sp.identity(p.cols)]).tocsr()
    _, _, passes, fallbacks = rs.restart_cycles(m, np.concatenate([p.b, np.zeros(p.cols)]), CYCLE,
                                                4, "fp16")
    assert passes == 4 * (CYCLE - 1) and fallbacks > passes // 4


@pytest.fixture(scope="module")
def amfls():
    import amfls_solver_gb300 as m

    m.load_library()
    return m


def on_gpu(amfls, p):
    from test_gpu_parity import csr_tensor

    return amfls.DeviceOperator(csr_tensor(p)), torch.from_numpy(p.b).cuda()


@pytest.mark.gpu
@pytest.mark.parametrize("storage", ["fp32", "fp16"])
def test_fallbacks_repeat_bit_for_bit(amfls, storage):
    op, b = on_gpu(amfls, problems.scaled_uniform_csr(**DEEP))
    opts = dict(reduced_basis=storage, maximum_depth=300, tolerance=1e-14)
    first = amfls.solve_amfls(op, b, **opts)
    assert first.reduced_basis_levels == 299 and first.reduced_basis_fallbacks > 100
    for _ in range(5):
        again = amfls.solve_amfls(op, b, **opts)
        assert (again.depth, again.reduced_basis_fallbacks) == (
            first.depth, first.reduced_basis_fallbacks)
        assert torch.equal(again.solution, first.solution)


@pytest.mark.gpu
def test_cycles_with_fallbacks_match_the_oracle(amfls):
    from test_gpu_parity import check_solution

    p = problems.scaled_uniform_csr(**CYCLES)
    op, b = on_gpu(amfls, p)
    tol = 1e-9
    r = amfls.run_amfls_mixed(op, b, values="fp64", reduced_basis="fp16", inner_tolerance=1e-14,
                              maximum_refinements=20, maximum_depth=CYCLE, regularization=REG,
                              tolerance=tol)
    assert r.status == 0 and r.reduced_basis_fallbacks > r.reduced_basis_levels // 4
    o = orc.solve_amfls(p, regularization=REG, tolerance=tol, seed=0)
    check_solution(p, r.solution.cpu().numpy(), np.asarray(o["solution"]), REG, tol, True)
