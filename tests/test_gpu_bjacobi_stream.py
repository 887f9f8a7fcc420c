"""The streamed block-Jacobi apply (one right-hand side, 32 MiB of inverses or more) against dense solves with the
operator's own diagonal blocks: blocks in two parts (105 x 105 in FP64) and whole, one to eight elements
per team with a partial last tile, FP64 and FP32 inverses and vectors, out of place and in place.

Tolerances as the other block-Jacobi tests: FP64 1e-10 of the largest entry, FP32 1e-4 in the 2-norm."""
import pytest
import torch

from cases import make_mesh, material, tandem_quadrature
from tandem_b200.operator import DGOperator, ELASTICITY, FP32, FP64, POISSON

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("kind,dim,n,N", [(ELASTICITY, 3, 7, 4), (ELASTICITY, 3, 10, 3), (ELASTICITY, 3, 17, 2),
                                          (ELASTICITY, 2, 139, 3), (POISSON, 2, 189, 4)])
def test_streamed_block_jacobi(kind, dim, n, N):
    op = DGOperator(make_mesh(dim, n, N, True), N, kind, tandem_quadrature(dim, N))
    op.set_material(*material(kind, dim, op.volume_coords(), True))
    bs = op.bs
    assert op.E * (((bs // 2 + 1) * bs + 3) // 4 * 4) * 4 >= 32 << 20  # bytes in FP32
    x = torch.randn(op.ndof, dtype=torch.float64, device=DEV, generator=torch.Generator(DEV).manual_seed(1))
    op.bjacobi_setup(FP64)
    blk = torch.as_tensor(op.bjacobi_blocks(), device=DEV)
    ref = torch.linalg.solve(blk, x.reshape(op.E, bs, 1)).reshape(-1)
    del blk
    for inv, prec, dt in ((FP64, FP64, torch.float64), (FP32, FP64, torch.float64), (FP32, FP32, torch.float32)):
        op.bjacobi_setup(inv)
        for inplace in (False, True):
            r = x.to(dt, copy=True)
            z = r if inplace else torch.full_like(r, 7.0)
            op.bjacobi_apply(r, z, prec)
            d = z.double() - ref
            if inv == FP64:
                assert d.abs().max() <= 1e-10 * ref.abs().max(), inplace
            else:
                assert d.norm() <= 1e-4 * ref.norm(), (prec, inplace)
