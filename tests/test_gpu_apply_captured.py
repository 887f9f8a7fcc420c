"""An apply replayed from a graph is no slower than one issued from the host: the facet kernel starts
behind the volume kernel there too.  (That its results stay in order under capture:
test_gpu_apply_warp.py, the overlapping kernels.)  The bound leaves 10 % for the spread of short
timings."""
import numpy as np
import pytest
import torch

from cases import make_mesh, material, tandem_quadrature
from tandem_b200.operator import DGOperator, ELASTICITY, FP32, FP64

pytestmark = pytest.mark.gpu


def device_us(f, reps, per):
    f()
    best = np.inf
    for _ in range(7):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        a.record()
        for _ in range(reps):
            f()
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b) / (reps * per) * 1e3)
    return best


@pytest.mark.parametrize("precision", [FP64, FP32])
def test_captured_apply_time(precision):
    op = DGOperator(make_mesh(3, 3, 4, True), 4, ELASTICITY, tandem_quadrature(3, 4))
    op.set_material(*material(ELASTICITY, 3, op.volume_coords(), True))
    op.set_apply_config(precision, "face")
    dt = torch.float64 if precision == FP64 else torch.float32
    x = torch.randn(op.ndof, dtype=dt, device="cuda")
    y = torch.empty_like(x)
    s = torch.cuda.Stream()
    issued = device_us(lambda: op.apply(x, y, precision), 40, 1)
    with torch.cuda.stream(s):
        op.apply(x, y, precision, stream=s)
        s.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            for _ in range(20):
                op.apply(x, y, precision, stream=s)
    assert device_us(graph.replay, 3, 20) <= 1.1 * issued
