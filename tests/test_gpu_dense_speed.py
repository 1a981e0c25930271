"""Dense products of few outputs (along the contiguous dimension) and of many
outputs with few chunks (across it) keep the GPU busy: both directions read the
same matrix, so the one does not take longer than the other.  Device times,
from products captured into a CUDA graph, the fastest of six replays."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def product_us(op, rows, cols, columns, reps=20):
    from amfls_solver_gb300 import _native

    x = torch.randn(cols * columns, dtype=torch.float64, device="cuda")
    y = torch.empty(rows * columns, dtype=torch.float64, device="cuda")
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    ptr = ctypes.c_void_p

    def run():
        _native.check(_native.load().amfls_gpu_operator_apply(
            op.handle, ptr(x.data_ptr()), columns, ptr(y.data_ptr()), ptr(stream.cuda_stream)))

    best = float("inf")
    with torch.cuda.stream(stream):
        for _ in range(3):
            run()
        stream.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            for _ in range(reps):
                run()
        for _ in range(6):
            start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            start.record(stream)
            graph.replay()
            end.record(stream)
            stream.synchronize()
            best = min(best, start.elapsed_time(end) * 1e3 / reps)
    return best


def both(rows, cols, columns):
    import amfls_solver_gb300 as amfls

    a = torch.randn(rows, cols, dtype=torch.float64, device="cuda")
    along = product_us(amfls.DeviceOperator(a), rows, cols, columns)
    return along, product_us(amfls.DeviceOperator(a.t().contiguous().t()), rows, cols, columns)


@pytest.mark.parametrize("rows,cols", [(40, 300), (120, 2000)])
@pytest.mark.parametrize("columns", [2, 3])
def test_few_outputs_along(rows, cols, columns):
    along, across = both(rows, cols, columns)
    assert along <= 1.15 * across


@pytest.mark.parametrize("rows", [8192, 16384])
def test_many_outputs_across(rows):
    along, across = both(rows, 512, 1)
    assert across <= 1.15 * along
