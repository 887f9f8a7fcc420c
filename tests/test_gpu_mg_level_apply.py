"""Level applies of the multigrid hierarchy on their own, every block size that the half-read form takes, against the
level's blocks: whole rows, and one block of every symmetric pair with the transposed product
gathered -- several elements per warp with a partial last warp (an odd number of elements), 2D and 3D, FP64
blocks and their FP32 copies, with and without a right-hand side.  And that the blocks are symmetric.

Tolerance: 1e-13 of the largest sum of |a||x| (at most 150 terms, summed in another order); symmetry 1e-11 of the
largest entry (rounding of the probing and the triple products)."""
import numpy as np
import pytest
import torch

from cases import material, tandem_quadrature
from tandem_b200 import mesh as M
from tandem_b200.operator import DGOperator, ELASTICITY, FP64, MIXED, POISSON

pytestmark = pytest.mark.gpu


def operator(kind, dim, n, N):
    m = M.square_mesh(n) if dim == 2 else M.cube_mesh(n)
    m = M.build(M.SimplexMesh(dim, m.vertices, m.elements[:-1]), N)
    op = DGOperator(m, N, kind, tandem_quadrature(dim, N))
    op.set_material(*material(kind, dim, op.volume_coords(), True))
    return op


def block_apply(A, nbr, x):
    """A x and |A| |x| with A given by rows of blocks, and both from the lower element's blocks alone."""
    E, NB, bs, _ = A.shape
    X = x.reshape(E, bs)
    whole, half, size = np.zeros((E, bs)), np.zeros((E, bs)), np.zeros((E, bs))
    for s in range(NB):
        e = np.nonzero(nbr[:, s] >= 0)[0]
        n = nbr[e, s]
        y = np.einsum("eij,ej->ei", A[e, s], X[n])
        whole[e] += y
        size[e] += np.einsum("eij,ej->ei", abs(A[e, s]), abs(X[n]))
        low = n >= e if s == 0 else n > e
        half[e[low]] += y[low]
        if s:
            np.add.at(half, n[low], np.einsum("eij,ei->ej", A[e, s][low], X[e[low]]))
    return whole.ravel(), half.ravel(), size.max()


@pytest.mark.parametrize("kind,dim,n,N", [(POISSON, 2, 4, 4), (ELASTICITY, 2, 4, 4), (POISSON, 3, 2, 4), (ELASTICITY, 3, 2, 4),
                                          (ELASTICITY, 3, 4, 2)])
@pytest.mark.parametrize("precision", [FP64, MIXED])
def test_level_apply(kind, dim, n, N, precision):
    op = operator(kind, dim, n, N)
    assert op.E % 2 == 1
    op.mg_setup(strategy="full", smooth_precision=precision)
    info = op.mg_info()
    taken = set()
    for level, bs in enumerate(info["block_sizes"][:-1]):
        A, nbr = op.mg_level_matrix(level)
        s = np.nonzero(nbr[:, 1] >= 0)[0]
        other = nbr[s, 1]
        back = np.argmax(nbr[other] == s[:, None], axis=1)
        assert np.abs(A[s, 1] - A[other, back].transpose(0, 2, 1)).max() <= 1e-11 * np.abs(A).max()
        if precision == MIXED:
            A = A.astype(np.float32).astype(np.float64)
        x = np.random.default_rng(level).standard_normal((2, op.E * bs))
        whole, half, size = block_apply(A, nbr, x[0])
        xd = torch.as_tensor(x, device="cuda")
        y = torch.empty_like(xd[0])
        for b in (None, xd[1]):
            sign, off = (1.0, 0.0) if b is None else (-1.0, x[1])
            op.mg_level_apply(level, xd[0], y, b)
            assert np.abs(y.cpu().numpy() - (off + sign * whole)).max() <= 1e-13 * size
            if bs in (6, 10, 12, 20, 30):
                taken.add(bs)
                op.mg_level_apply(level, xd[0], y.fill_(7.0), b, half=True)
                assert np.abs(y.cpu().numpy() - (off + sign * half)).max() <= 1e-13 * size
    assert taken
