"""The continuous P1 level's apply and restriction share a row among 8, 4, 2 or 1 lanes, as the rows of all columns
fill the GPU: a V-cycle of 1, 4, 8 and 16 columns (10,201 vertices, 8 to 1 lanes) gives every column what it
gets alone.

Tolerance: 1e-8 of the largest entry -- rounding in another order, through the coarse CG's some hundred
iterations on a system of condition 1e4 to 1e5 (1e-16 x 1e2 x 1e5, with room)."""
import pytest
import torch

from cases import make_mesh, material, tandem_quadrature
from tandem_b200.operator import DGOperator, ELASTICITY, POISSON

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n", [(POISSON, 100), (ELASTICITY, 70)])
def test_columns_agree_over_the_lane_counts(kind, n):
    op = DGOperator(make_mesh(2, n, 2, True), 2, kind, tandem_quadrature(2, 2))
    op.set_material(*material(kind, 2, op.volume_coords(), True))
    op.mg_setup(smooth_its=4)
    R = torch.randn(16, op.ndof, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(2))
    alone = torch.empty_like(R)
    for i in range(16):
        op.mg_apply(R[i], alone[i])
    for nrhs in (4, 8, 16):
        Z = torch.empty_like(R[:nrhs])
        op.mg_apply(R[:nrhs], Z, nrhs=nrhs)
        assert (Z - alone[:nrhs]).abs().max() <= 1e-8 * alone.abs().max()
