"""A new material drops the device data of both precisions, the kernels' status words among it: a solve in one
precision after the other has run reads none that is gone."""
import numpy as np
import pytest
import torch

from cases import make_mesh, material, tandem_quadrature
from oracle import Oracle
from tandem_b200.operator import DGOperator, ELASTICITY, FP32, FP64

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("update", [False, True])
@pytest.mark.parametrize("first", [FP64, FP32])
def test_solve_after_the_other_precision_and_a_new_material(first, update):
    m, q = make_mesh(3, 2, 2, True), tandem_quadrature(3, 2)
    op, orc = DGOperator(m, 2, ELASTICITY, q), Oracle(m, 2, ELASTICITY, q)
    c0, c1 = material(ELASTICITY, 3, op.volume_coords(), True)
    op.set_material(c0, c1)
    second = FP32 if first == FP64 else FP64
    x = torch.randn(op.ndof, dtype=torch.float64, device=DEV)
    op.bjacobi_setup(second)  # kept by update_material
    xf = x.to(torch.float32 if first == FP32 else torch.float64)
    op.apply(xf, torch.empty_like(xf), first)
    (op.update_material if update else op.set_material)(1.1 * c0, 1.1 * c1)
    orc.set_material(1.1 * c0, 1.1 * c1)
    if not update:
        op.bjacobi_setup(second)
    u = torch.randn(op.ndof, dtype=torch.float64, device=DEV)
    b = torch.as_tensor(orc.apply(u.cpu().numpy()), device=DEV)
    x = torch.zeros_like(b)
    st = op.solve(b, x, precision=second, rtol=1e-10 if second == FP64 else 1e-6)
    res = b.cpu().numpy() - orc.apply(x.cpu().numpy())
    assert st["converged"] and np.linalg.norm(res) <= (1.01e-10 if second == FP64 else 1.01e-6) * np.linalg.norm(b.cpu().numpy())
