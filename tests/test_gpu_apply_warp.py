"""The warp-tile FP64 apply (families face / face2) against the oracle where its tiling changes: partial
tiles of 8 elements and facets, points in full and half blocks (conical and tandem rules), tables in
shared memory and through L1 (3D p4 with conical rules), work items shared by several warps (small
meshes, the last round of larger ones), CTA sizes, and many right-hand sides at a padded stride.

Tolerance: 1e-12 of the largest entry, as every FP64 kernel against the oracle (summation order)."""
import numpy as np
import pytest
import torch

from cases import make_mesh, material, tandem_quadrature
from oracle import Oracle
from tandem_b200.operator import DGOperator, ELASTICITY, FP64, POISSON, Quadrature

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

CASES = [  # kind, dim, n, degree, rule
    (ELASTICITY, 3, 1, 4, "conical"), (ELASTICITY, 3, 3, 4, "tandem"), (ELASTICITY, 3, 7, 4, "tandem"),
    (ELASTICITY, 3, 12, 4, "tandem"), (ELASTICITY, 3, 8, 3, "conical"), (ELASTICITY, 3, 3, 3, "tandem"),
    (ELASTICITY, 3, 5, 2, "conical"), (ELASTICITY, 3, 3, 1, "tandem"), (ELASTICITY, 3, 3, 1, "conical"),
    (POISSON, 3, 3, 4, "conical"), (POISSON, 3, 7, 4, "tandem"), (POISSON, 3, 5, 3, "conical"),
    (POISSON, 3, 3, 2, "tandem"), (POISSON, 3, 3, 1, "tandem"),
    (POISSON, 2, 1, 4, "tandem"), (POISSON, 2, 9, 4, "conical"), (POISSON, 2, 5, 3, "tandem"),
    (POISSON, 2, 5, 2, "conical"), (POISSON, 2, 40, 1, "tandem"),
    (ELASTICITY, 2, 7, 4, "conical"), (ELASTICITY, 2, 5, 3, "conical"), (ELASTICITY, 2, 5, 2, "tandem"),
    (ELASTICITY, 2, 1, 1, "tandem"),
]


def problem(kind, dim, n, N, rule):
    m = make_mesh(dim, n, N, True)
    q = tandem_quadrature(dim, N) if rule == "tandem" else Quadrature.conical(dim, 2 * N + 1)
    op, orc = DGOperator(m, N, kind, q), Oracle(m, N, kind, q)
    c = material(kind, dim, op.volume_coords(), True)
    op.set_material(*c)
    orc.set_material(*c)
    return op, orc


@pytest.mark.parametrize("case", CASES, ids=lambda c: "k{}d{}n{}p{}{}".format(*c))
def test_warp_tile_apply_matches_oracle(case):
    op, orc = problem(*case)
    x = np.random.default_rng(5).standard_normal(op.ndof)
    ref = orc.apply(x)
    xd = torch.as_tensor(x, device=DEV)
    for ctas in (0, 1, 2, 3, 4):
        op.set_apply_config(FP64, "face2", ctas)
        y = torch.full((op.ndof,), 3.0, dtype=torch.float64, device=DEV)
        op.apply(xd, y)
        assert np.abs(y.cpu().numpy() - ref).max() <= 1e-12 * np.abs(ref).max(), ctas


@pytest.mark.parametrize("kind,dim,n,N,nrhs", [(POISSON, 2, 9, 4, 11), (ELASTICITY, 2, 6, 3, 8), (ELASTICITY, 3, 2, 4, 9)])
def test_warp_tile_apply_columns(kind, dim, n, N, nrhs):
    op, orc = problem(kind, dim, n, N, "tandem")
    op.set_apply_config(FP64, "face2")
    ld = op.ndof + 5
    X = torch.randn(nrhs, ld, dtype=torch.float64, device=DEV)
    Y = torch.full((nrhs, ld), 7.0, dtype=torch.float64, device=DEV)
    op.apply(X, Y, nrhs=nrhs, ld=ld)
    for r in range(nrhs):
        ref = orc.apply(X[r, :op.ndof].cpu().numpy())
        assert np.abs(Y[r, :op.ndof].cpu().numpy() - ref).max() <= 1e-12 * np.abs(ref).max()
        assert torch.all(Y[r, op.ndof:] == 7.0)


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("kind,dim,n,N", [(POISSON, 2, 4, 2), (ELASTICITY, 3, 4, 2), (ELASTICITY, 3, 9, 4)])
def test_overlapping_volume_and_facet_kernels_keep_their_order(kind, dim, n, N, captured):
    """The facet kernel starts while the volume kernel runs.  A chain x -> A x -> A A x (each apply reads
    what the one before it wrote, scaled by a kernel between them) gives what separate applies give."""
    op, orc = problem(kind, dim, n, N, "tandem")
    op.set_apply_config(FP64, "face")
    x0 = torch.randn(op.ndof, dtype=torch.float64, device=DEV)
    x, y = x0.clone(), torch.empty_like(x0)
    s = torch.cuda.Stream()

    def chain():
        for _ in range(6):
            op.apply(x, y, stream=s)
            torch.mul(y, scale, out=x)

    scale = 1.0 / np.abs(orc.apply(x0.cpu().numpy())).max()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        if captured:
            graph = torch.cuda.CUDAGraph()
            op.apply(x, y, stream=s)
            s.synchronize()
            with torch.cuda.graph(graph, stream=s):
                chain()
            graph.replay()
        else:
            chain()
    s.synchronize()
    ref = x0.cpu().numpy()
    for _ in range(6):
        ref = orc.apply(ref) * scale
    # 1e-12 from each of the six applies, with room for what the chain makes of the first ones'
    assert np.abs(x.cpu().numpy() - ref).max() <= 1e-10 * np.abs(ref).max()
