"""The warp-tile FP32 apply (families face / face2 / tc05) against the oracle where its tiling changes:
partial tiles of 16 elements and facets, points in full and half blocks, tables in shared memory and
through L1, work items shared by several warps, CTA sizes, many right-hand sides at a padded stride;
FP32 vectors, FP64 vectors (mixed) and the single TF32 pass; and what the tuner may pick.

Tolerance: 2e-5 of the largest entry, as every FP32 kernel against the oracle.  The single TF32 pass
rounds both factors of four chained products (values, gradients, their lift-backs) to 2^-11: 4e-3."""
import numpy as np
import pytest
import torch

from cases import make_mesh, material, tandem_quadrature
from oracle import Oracle
from tandem_b200.operator import DGOperator, ELASTICITY, FP32, MIXED, POISSON, Quadrature, TF32

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

CASES = [  # kind, dim, n, degree, rule
    (ELASTICITY, 3, 1, 4, "conical"), (ELASTICITY, 3, 3, 4, "tandem"), (ELASTICITY, 3, 9, 4, "tandem"),
    (ELASTICITY, 3, 6, 3, "conical"), (ELASTICITY, 3, 3, 3, "tandem"), (ELASTICITY, 3, 5, 2, "conical"),
    (ELASTICITY, 3, 3, 1, "tandem"), (POISSON, 3, 3, 4, "conical"), (POISSON, 3, 7, 4, "tandem"),
    (POISSON, 3, 5, 3, "conical"), (POISSON, 3, 3, 2, "tandem"), (POISSON, 3, 3, 1, "tandem"),
    (POISSON, 2, 1, 4, "tandem"), (POISSON, 2, 9, 4, "conical"), (POISSON, 2, 5, 3, "tandem"),
    (POISSON, 2, 40, 1, "tandem"), (ELASTICITY, 2, 7, 4, "conical"), (ELASTICITY, 2, 5, 3, "conical"),
    (ELASTICITY, 2, 5, 2, "tandem"), (ELASTICITY, 2, 1, 1, "tandem"),
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
def test_warp_tile_fp32_apply_matches_oracle(case):
    op, orc = problem(*case)
    x = np.random.default_rng(5).standard_normal(op.ndof)
    ref = orc.apply(x)
    for prec, tol in ((FP32, 2e-5), (MIXED, 2e-5), (TF32, 4e-3)):
        xd = torch.as_tensor(x, device=DEV, dtype=torch.float32 if prec == FP32 else torch.float64)
        for family, ctas in (("face", 0), ("face2", 1), ("face", 3), ("tc05", 0)):
            op.set_apply_config(FP32, family, ctas)
            y = torch.full_like(xd, 3.0)
            op.apply(xd, y, precision=prec)
            assert np.abs(y.double().cpu().numpy() - ref).max() <= tol * np.abs(ref).max(), (prec, family, ctas)


@pytest.mark.parametrize("kind,dim,n,N,nrhs", [(POISSON, 2, 9, 4, 11), (ELASTICITY, 3, 2, 4, 9)])
def test_warp_tile_fp32_apply_columns(kind, dim, n, N, nrhs):
    op, orc = problem(kind, dim, n, N, "tandem")
    op.set_apply_config(FP32, "face")
    ld = op.ndof + 5  # an odd stride: no column but the first starts on a 16-byte boundary
    X = torch.randn(nrhs, ld, dtype=torch.float32, device=DEV)
    Y = torch.full((nrhs, ld), 7.0, dtype=torch.float32, device=DEV)
    op.apply(X, Y, precision=FP32, nrhs=nrhs, ld=ld)
    for r in range(nrhs):
        ref = orc.apply(X[r, :op.ndof].double().cpu().numpy())
        assert np.abs(Y[r, :op.ndof].double().cpu().numpy() - ref).max() <= 2e-5 * np.abs(ref).max()
        assert torch.all(Y[r, op.ndof:] == 7.0)


def test_tuner_keeps_the_accurate_kernel_on_small_shapes():
    """2D degree-1 Poisson: the SIMT kernel beats the element-centric one severalfold, so it stays."""
    op, _ = problem(POISSON, 2, 40, 1, "tandem")
    ms = {}
    for t in op.autotune(FP32):
        ms[t["family"]] = min(t["ms"], ms.get(t["family"], 1e9))
    x = torch.randn(op.ndof, dtype=torch.float32, device=DEV)
    tuned, simt = torch.empty_like(x), torch.empty_like(x)
    op.apply(x, tuned, precision=FP32)
    op.set_apply_config(FP32, "simt")
    op.apply(x, simt, precision=FP32)
    if ms["simt"] < 0.95 * ms["tensor"]:
        assert torch.equal(tuned, simt)
