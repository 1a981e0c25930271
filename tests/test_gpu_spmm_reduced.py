"""GPU tests of CSR block products on reduced values bit by bit: a row of at
most 64 nonzeros is one chain of FP32 multiply-adds in storage order, however
its length compares with its neighbours' (blocks whose FP64 products share long
rows out among all lanes are among the cases)."""
import numpy as np
import pytest
import torch

from test_gpu_parity import csr_tensor
from test_gpu_resident import ragged_csr

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def amfls():
    import amfls_solver_gb300 as m

    m.load_library()
    return m


def fp32_chains(mat, x):
    """Row sums as chains of FP32 multiply-adds.  The product of two FP32
    numbers is exact in the long double sum, whose rounding lies at least 2^-40
    of a unit below FP32's."""
    out = np.empty((mat.shape[0], x.shape[1]), dtype=np.float32)
    wide = x.astype(np.longdouble)
    for i, row in enumerate(mat):
        acc = np.zeros(x.shape[1], dtype=np.float32)
        for j in np.flatnonzero(row):
            acc = (np.longdouble(row[j]) * wide[j] + acc.astype(np.longdouble)).astype(np.float32)
        out[i] = acc
    return out


@pytest.mark.parametrize("values", ["fp32", "bf16"])
@pytest.mark.parametrize("lengths", [[33], [1, 1, 1, 1, 24], [8, 9, 0, 17], [1, 64, 2, 63], [20]])
def test_rows_are_fp32_chains(amfls, lengths, values):
    p = ragged_csr(307, 900, lengths, seed=len(lengths))
    a = p.to_dense()
    assert max(np.count_nonzero(a, axis=0).max(), np.count_nonzero(a, axis=1).max()) <= 64
    cast = torch.float32 if values == "fp32" else torch.bfloat16
    reduced = torch.from_numpy(a).to(cast).to(torch.float32).numpy()
    op = amfls.DeviceOperator(csr_tensor(p)).reduced(values)
    rng = np.random.default_rng(4)
    for transpose, mat in ((False, reduced), (True, reduced.T)):
        x = rng.standard_normal((mat.shape[1], 8))
        want = fp32_chains(mat, x.astype(np.float32))
        for s in (2, 3, 4, 7, 8):
            y = op.apply(torch.from_numpy(x[:, :s].copy()).cuda(), transpose=transpose)
            assert np.array_equal(y.cpu().numpy().astype(np.float32), want[:, :s])
