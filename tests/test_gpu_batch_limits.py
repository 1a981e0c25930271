"""How many problems of a batch run at a time.  A problem's seconds begin when a
worker takes it, so their sum over the batch's wall time is the mean number in
flight: at most eight CSR problems, whatever else the batch holds, and more
where the process asks for more hardware queues."""
import json
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]

SCRIPT = """
import json, sys
import numpy as np, torch
import amfls_solver_gb300 as amfls
from amfls_solver_gb300 import problems
sys.path.insert(0, "tests")
from test_gpu_parity import _matrix_tensor, csr_tensor

csr, dense, workers = (int(v) for v in sys.argv[1:])
probs = [problems.scaled_uniform_csr(3000, 700, per_row=8, decades=3.0, noise=1e-6, seed=i)
         for i in range(csr)]
mats = [(amfls.DeviceOperator(csr_tensor(p)), torch.from_numpy(p.b).cuda()) for p in probs]
for i in range(dense):
    p = problems.scaled_dense(900, 60, decades=2.0, seed=i)
    mats.append((amfls.DeviceOperator(_matrix_tensor(p)), torch.from_numpy(p.b).cuda()))
opts = dict(regularization=1e-3, tolerance=1e-9)
amfls.run_amfls_batch(mats, workers=workers, **opts)
results, seconds, wall = amfls.run_amfls_batch(mats, workers=workers, **opts)
same = []
for (op, b), r in zip(mats, results):
    one = amfls.solve_amfls(op, b, **opts)
    # both lie within tol of the solution in the energy norm
    bound = 2 * opts["tolerance"] * op.validation_error_model()[0] / opts["regularization"] ** 0.5
    same.append(r.status == one.status == 0 and float(torch.linalg.norm(r.solution - one.solution))
                <= 2 * bound * float(torch.linalg.norm(one.solution)))
print(json.dumps(dict(same=same, csr=float(np.sum(seconds[:csr])) / wall,
                      dense=float(np.sum(seconds[csr:])) / wall)))
"""


def batch(csr, dense, workers, connections=None):
    env = {k: v for k, v in os.environ.items() if k != "CUDA_DEVICE_MAX_CONNECTIONS"}
    if connections is not None:
        env["CUDA_DEVICE_MAX_CONNECTIONS"] = str(connections)
    run = subprocess.run([sys.executable, "-W", "ignore", "-c", SCRIPT, str(csr), str(dense),
                          str(workers)], cwd=ROOT, env=env, capture_output=True, text=True,
                         timeout=300)
    assert run.returncode == 0, run.stderr
    out = json.loads(run.stdout.strip().splitlines()[-1])
    assert all(out["same"])
    return out


@pytest.mark.parametrize("dense", [0, 1, 5])
def test_eight_csr_problems_at_a_time(dense):
    assert batch(24, dense, 24 + dense)["csr"] <= 8.0


def test_more_where_the_process_asks_for_more_queues():
    assert 8.0 < batch(32, 0, 16, connections=16)["csr"] <= 16.0


@pytest.mark.parametrize("csr,dense", [(1, 0), (0, 3), (2, 3)])
def test_small_and_mixed_batches(csr, dense):
    batch(csr, dense, 4)
