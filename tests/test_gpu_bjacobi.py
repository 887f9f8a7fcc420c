"""Block-Jacobi apply with the packed symmetric inverses against dense solves with the oracle's
diagonal blocks: odd and even block sizes, one right-hand side (rows) and several (tensor pipe, partial
groups of 8 and of 32 columns, padded stride), FP64 vectors with FP64 and FP32 inverses, FP32 vectors,
in place.

Tolerances: FP64 1e-10 of the largest entry (the dense solve's own conditioning, as the
single-column test); FP32 inverses or vectors 1e-4 in the 2-norm."""
import numpy as np
import pytest
import torch

from cases import product_and_oracle
from tandem_b200.operator import ELASTICITY, FP32, FP64, POISSON

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("kind,dim,n,N", [(POISSON, 2, 5, 4), (POISSON, 2, 3, 1), (POISSON, 3, 2, 2), (POISSON, 3, 1, 4),
                                          (ELASTICITY, 2, 5, 4), (ELASTICITY, 2, 3, 1), (ELASTICITY, 3, 1, 1),
                                          (ELASTICITY, 3, 1, 3), (ELASTICITY, 3, 1, 4)])
@pytest.mark.parametrize("nrhs", [1, 2, 9, 33])
def test_packed_block_jacobi(kind, dim, n, N, nrhs):
    _, op, orc = product_and_oracle(kind, dim, n, N, True, True)
    blk = orc.assemble_diag()
    ld = op.ndof + 3
    R = np.random.default_rng(4).standard_normal((nrhs, ld))
    ref = np.stack([np.linalg.solve(blk, r[:op.ndof].reshape(op.E, op.bs, 1)).reshape(-1) for r in R])
    scale = np.abs(ref).max()

    def run(inv, prec, dt, inplace=False):
        op.bjacobi_setup(inv)
        r = torch.as_tensor(R, dtype=dt, device=DEV).contiguous()
        z = r if inplace else torch.full_like(r, 7.0)
        op.bjacobi_apply(r, z, prec, nrhs=nrhs, ld=ld)
        if not inplace:
            assert torch.all(z[:, op.ndof:] == 7.0)
        return z[:, :op.ndof].double().cpu().numpy()

    for inplace in (False, True):
        assert np.abs(run(FP64, FP64, torch.float64, inplace) - ref).max() <= 1e-10 * scale
    for prec, dt in ((FP64, torch.float64), (FP32, torch.float32)):
        assert np.linalg.norm(run(FP32, prec, dt) - ref) <= 1e-4 * np.linalg.norm(ref)
