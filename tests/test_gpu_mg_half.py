"""Level applies of multigrid levels larger than L2: one right-hand side reads each symmetric pair of
off-diagonal blocks once (3D elasticity p4 -> p2 blocks of 30, from 2,800 elements in FP64 and twice that
in FP32), several right-hand sides read whole block rows.  One V-cycle of a column alone and among
two columns differs by the order of summation only: 1e-11 of the largest entry (rounding times the
cycle's 24 level applies; the coarse CG takes the same iterations)."""
import pytest
import torch

from cases import make_mesh, material, tandem_quadrature
from tandem_b200.operator import DGOperator, ELASTICITY, FP32, FP64, MIXED, POISSON

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n,precision", [(ELASTICITY, 8, FP64), (ELASTICITY, 10, MIXED), (POISSON, 14, FP64)])
def test_half_read_level_apply(kind, n, precision):
    m = make_mesh(3, n, 4, True)
    op = DGOperator(m, 4, kind, tandem_quadrature(3, 4))
    op.set_material(*material(kind, 3, op.volume_coords(), True))
    op.mg_setup(smooth_its=6, smooth_precision=precision)
    g = torch.Generator(device="cuda").manual_seed(2)
    R = torch.randn(2, op.ndof, dtype=torch.float64, device="cuda", generator=g)
    Z = torch.empty_like(R)
    op.mg_apply(R, Z, nrhs=2)
    z = torch.empty_like(R[0])
    for i in range(2):
        op.mg_apply(R[i].contiguous(), z)
        assert (z - Z[i]).abs().max() <= 1e-11 * Z[i].abs().max()
