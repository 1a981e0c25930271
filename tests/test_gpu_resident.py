"""GPU tests of the resident level kernel (whole checkpoint intervals of CSR
solves as one cooperative kernel) where it can go wrong: bases narrower than a
panel and at its edges, fewer rows than blocks, row groups and units that end
inside a warp, rows of every lane count of the sliced tables, empty rows, wide
problems, and solves that share the GPU.  Status, stop reason, depth and basis
rank must be the oracle's, and x must pass the checks of the parity tests."""
import threading

import numpy as np
import pytest
import torch

from oracle import amfls_oracle as orc
from test_gpu_parity import check_solution, csr_tensor

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def amfls():
    import amfls_solver_gb300 as m

    m.load_library()
    return m


def ragged_csr(rows, cols, lengths, seed):
    """Rows of the given lengths (taken in turn) at distinct columns."""
    from amfls_solver_gb300 import problems

    rng = np.random.default_rng(seed)
    lens = np.minimum(np.resize(lengths, rows), cols)
    rng.shuffle(lens)
    col = np.concatenate([np.sort(rng.choice(cols, n, replace=False)) for n in lens])
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    p = problems.CsrProblem(rows, cols, off, col.astype(np.int64),
                            rng.standard_normal(col.size), np.zeros(rows))
    p.b = p.matvec(rng.standard_normal(cols)) + 1e-3 * rng.standard_normal(rows)
    return p


SIZES = [
    (40, 1, [1]), (50, 17, [0, 3, 5]), (90, 31, [4]), (90, 32, [4]), (90, 33, [4]),
    (200, 64, [7, 9]), (200, 65, [8, 0, 17]), (150, 97, [1, 2, 3, 97]),
    (700, 152, [8, 9, 16, 17]), (900, 305, [5, 33, 64, 65]), (60, 200, [12]),
    (1500, 640, [2, 8, 128, 129, 256, 257, 600]),
]


@pytest.mark.parametrize("reg", [0.0, 1e-2])
@pytest.mark.parametrize("rows,cols,lengths", SIZES)
def test_resident_solve_matches_oracle(amfls, rows, cols, lengths, reg):
    p = ragged_csr(rows, cols, lengths, seed=rows + cols)
    tol = 1e-8
    r = amfls.run_amfls(csr_tensor(p), torch.from_numpy(p.b).cuda(), regularization=reg,
                        tolerance=tol, seed=3)
    o = orc.solve_amfls(p, regularization=reg, tolerance=tol, seed=3)
    assert (r.status, r.stop_reason) == (o["status"], o["stop_reason"])
    assert r.depth == int(o["counters"][9]) and r.basis_rank == int(o["counters"][11])
    check_solution(p, r.solution.cpu().numpy(), np.asarray(o["solution"]), reg, tol,
                   r.status == 0)


@pytest.mark.parametrize("basis", ["fp32", "fp16"])
@pytest.mark.parametrize("rows,cols", [(300, 65), (2100, 513), (9000, 2050)])
def test_resident_reduced_sweeps(amfls, rows, cols, basis):
    """Restart cycles on the augmented operator with the reduced copy: certified
    at the tolerance, x within 2.5 tol of the FP64 oracle's in the energy norm."""
    from amfls_solver_gb300 import problems

    p = problems.scaled_uniform_csr(rows, cols, per_row=9, decades=1.0, noise=1e-6, seed=rows)
    reg, tol = 1e-2, 1e-9
    r = amfls.run_amfls_mixed(csr_tensor(p), torch.from_numpy(p.b).cuda(), values="fp64",
                              reduced_basis=basis, inner_tolerance=1e-14,
                              maximum_refinements=60, maximum_depth=100, regularization=reg,
                              tolerance=tol)
    assert r.status == 0 and r.reduced_basis_levels > 0
    o = orc.solve_amfls(p, regularization=reg, tolerance=tol, seed=0)
    check_solution(p, r.solution.cpu().numpy(), np.asarray(o["solution"]), reg, tol, True)


def test_resident_solves_share_the_gpu(amfls):
    """Solves on several threads and streams: the same bits as one at a time."""
    probs = [ragged_csr(800 + 37 * i, 200 + 11 * i, [6, 12], seed=i) for i in range(4)]
    data = [(amfls.DeviceOperator(csr_tensor(p)), torch.from_numpy(p.b).cuda()) for p in probs]
    alone = [amfls.solve_amfls(a, b, regularization=1e-2, tolerance=1e-9) for a, b in data]
    torch.cuda.synchronize()
    got = [None] * len(data)

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(3):
                got[i] = amfls.solve_amfls(data[i][0], data[i][1], regularization=1e-2,
                                           tolerance=1e-9)
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(data))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, g in zip(alone, got):
        assert g.depth == a.depth and torch.equal(g.solution, a.solution)
