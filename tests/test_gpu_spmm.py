"""GPU tests of CSR block products where rows of one block differ in length:
lengths at the edges of the split (8 and 9), of the row blocks (64 and 65) and of
the 64-element steps of longer rows, empty rows, two to nine columns, both
directions, FP64 and reduced values, against numpy."""
import numpy as np
import pytest
import torch

from test_gpu_parity import csr_tensor
from test_gpu_resident import ragged_csr

pytestmark = pytest.mark.gpu

LENGTHS = [[1, 1, 1, 1, 24], [8, 9, 0, 17], [1, 64, 2, 65, 63], [20], [80, 81, 127, 128, 129],
           [3, 1100, 0, 40], [1, 2, 3, 4, 5, 6, 7, 30]]


@pytest.fixture(scope="module")
def amfls():
    import amfls_solver_gb300 as m

    m.load_library()
    return m


@pytest.mark.parametrize("values,unit", [("fp64", 2.0 ** -53), ("fp32", 2.0 ** -24)])
@pytest.mark.parametrize("lengths", LENGTHS)
def test_block_products_match_numpy(amfls, lengths, values, unit):
    """|y - y_numpy| within both sides' rounding: n products summed with a
    relative error of at most n u each, and for reduced values the rounding of
    value and x: 2 (n + 3) u |A| |x|."""
    p = ragged_csr(611, 1200, lengths, seed=len(lengths))
    a = p.to_dense()
    op = amfls.DeviceOperator(csr_tensor(p))
    if values != "fp64":
        op = op.reduced(values)
    rng = np.random.default_rng(1)
    for s in range(2, 10):
        for transpose, mat in ((False, a), (True, a.T)):
            x = rng.standard_normal((mat.shape[1], s))
            y = op.apply(torch.from_numpy(x).cuda(), transpose=transpose).cpu().numpy()
            n = np.max(np.count_nonzero(mat, axis=1))
            bound = 2 * (n + 3) * unit * (np.abs(mat) @ np.abs(x))
            assert np.all(np.abs(y - mat @ x) <= bound)
