"""Block-Jacobi apply to several columns, by each route of its dispatch: every column apart (all rows fit
beside each other), rows in groups of two to five columns, the FP64 tensor pipe with one warp per element and with
four.  Checked against dense solves with the operator's own diagonal blocks, in place and at a
padded stride, with partial groups.  And the time: columns together never cost much more than one by one.

Tolerances as the other block-Jacobi tests: FP64 1e-10 of the largest entry, FP32 1e-4 in the 2-norm."""
import numpy as np
import pytest
import torch

from cases import make_mesh, material, tandem_quadrature
from tandem_b200.operator import DGOperator, ELASTICITY, FP32, FP64, POISSON

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def operator(kind, dim, n, N):
    op = DGOperator(make_mesh(dim, n, N, True), N, kind, tandem_quadrature(dim, N))
    op.set_material(*material(kind, dim, op.volume_coords(), True))
    return op


def solve_blocks(op, R):
    blk = torch.as_tensor(op.bjacobi_blocks(), device=DEV)
    r = R[:, :op.ndof].reshape(R.shape[0], op.E, op.bs).permute(1, 2, 0)
    return torch.linalg.solve(blk, r).permute(2, 0, 1).reshape(R.shape[0], -1)


# elements enough that two columns of rows no longer fit beside each other, and a few
@pytest.mark.parametrize("kind,dim,N,sizes", [
    (POISSON, 2, 3, (4, 64)), (ELASTICITY, 2, 2, (4, 58)), (POISSON, 2, 4, (3, 51)), (POISSON, 3, 3, (2, 11)),
    (ELASTICITY, 3, 2, (2, 9)), (POISSON, 3, 4, (2, 8)), (ELASTICITY, 3, 3, (1, 7)), (ELASTICITY, 3, 4, (1, 5))])
def test_columns_by_every_route(kind, dim, N, sizes):
    for n in sizes:
        op = operator(kind, dim, n, N)
        ld = op.ndof + 3
        X = torch.randn(33, ld, dtype=torch.float64, device=DEV, generator=torch.Generator(DEV).manual_seed(n))
        op.bjacobi_setup(FP64)
        ref = solve_blocks(op, X)
        for inv, prec, dt in ((FP64, FP64, torch.float64), (FP32, FP64, torch.float64), (FP32, FP32, torch.float32)):
            op.bjacobi_setup(inv)
            for nrhs in (2, 3, 4, 5, 6, 9, 33):
                for inplace in (False, True):
                    r = X[:nrhs].to(dt, copy=True)
                    z = r if inplace else torch.full_like(r, 7.0)
                    pad = r[:, op.ndof:].clone() if inplace else z[:, op.ndof:].clone()
                    op.bjacobi_apply(r, z, prec, nrhs=nrhs, ld=ld)
                    assert torch.equal(z[:, op.ndof:], pad)
                    d = z[:, :op.ndof].double() - ref[:nrhs]
                    if inv == FP64:
                        assert d.abs().max() <= 1e-10 * ref[:nrhs].abs().max(), (n, nrhs, inplace)
                    else:
                        assert d.norm() <= 1e-4 * ref[:nrhs].norm(), (n, inv, prec, nrhs, inplace)


def device_us(f, reps=30):
    f()
    best = np.inf
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        a.record()
        for _ in range(reps):
            f()
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b) / reps * 1e3)
    return best


@pytest.mark.parametrize("kind,dim,n,N", [(ELASTICITY, 3, 2, 4), (ELASTICITY, 3, 8, 4), (POISSON, 3, 10, 4),
                                          (ELASTICITY, 2, 60, 4)])
@pytest.mark.parametrize("inv", [FP64, FP32])
def test_two_columns_cost_at_most_two_applies(kind, dim, n, N, inv):
    op = operator(kind, dim, n, N)
    op.bjacobi_setup(inv)
    r = torch.randn(2, op.ndof, dtype=torch.float64, device=DEV)
    z = torch.empty_like(r)
    one = device_us(lambda: op.bjacobi_apply(r, z))
    # the bound leaves half an apply of room for the spread of short timings
    assert device_us(lambda: op.bjacobi_apply(r, z, nrhs=2)) <= 2.5 * one
