"""What the tuner keeps.  FP64: the configuration it measured as the fastest on the device, also where a call
takes less device time than the host needs to issue it (the solves replay it from graphs)."""
import pytest
import torch

from cases import make_mesh, material, tandem_quadrature
from tandem_b200 import _ffi
from tandem_b200.operator import DGOperator, ELASTICITY, FAMILIES, FP32, FP64, MIXED, POISSON, TF32

pytestmark = pytest.mark.gpu


def operator(kind, dim, n, N):
    op = DGOperator(make_mesh(dim, n, N, True), N, kind, tandem_quadrature(dim, N))
    op.set_material(*material(kind, dim, op.volume_coords(), True))
    return op


@pytest.mark.parametrize("kind,dim,n,N", [(POISSON, 2, 9, 1), (POISSON, 2, 9, 3), (ELASTICITY, 2, 9, 2),
                                          (POISSON, 3, 3, 2), (ELASTICITY, 3, 6, 3)])
def test_tuner_keeps_the_fastest_fp64_configuration(kind, dim, n, N):
    op = operator(kind, dim, n, N)
    assert op.apply_config(FP64) == dict(family="tensor", ctas_per_sm=0, tile=0)
    for nrhs in (1, 3):
        entries = op.autotune(FP64, nrhs=nrhs)
        best = min(entries, key=lambda e: e["ms"])
        assert op.apply_config(FP64) == {k: best[k] for k in ("family", "ctas_per_sm", "tile")}


def test_call_configuration_serves_single_applies_only():
    """tdg_set_call_config: single applies take it (the SIMT kernel repeats bit for bit), applies captured in a graph
    and the reported configuration do not; setting a configuration takes it back."""
    op = operator(ELASTICITY, 2, 9, 3)
    x = torch.randn(op.ndof, dtype=torch.float32, device="cuda")
    simt, y = torch.empty_like(x), torch.empty_like(x)
    op.set_apply_config(FP32, "simt")
    op.apply(x, simt, FP32)
    op.set_apply_config(FP32, "face")
    _ffi.check(_ffi.lib().tdg_set_call_config(op._h, FP32, FAMILIES.index("simt"), 0))
    assert op.apply_config(FP32)["family"] == "face"
    op.apply(x, y, FP32)
    assert torch.equal(y, simt)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            op.apply(x, y, FP32, stream=s)
    graph.replay()
    assert not torch.equal(y, simt) and (y - simt).abs().max() <= 4e-5 * simt.abs().max()
    op.set_apply_config(FP32, "face")
    op.apply(x, y, FP32)
    assert not torch.equal(y, simt)
    with pytest.raises(_ffi.TdgError, match="bad argument"):
        _ffi.check(_ffi.lib().tdg_set_call_config(op._h, FP64, 4, 0))


@pytest.mark.parametrize("kind,dim,n,N,nrhs,simt", [
    (POISSON, 2, 3, 1, 1, True), (POISSON, 2, 40, 1, 2, True), (POISSON, 3, 2, 1, 1, True),
    (POISSON, 2, 77, 2, 1, False), (POISSON, 2, 78, 2, 1, True), (POISSON, 2, 9, 2, 75, True),
    (POISSON, 2, 64, 3, 1, False), (POISSON, 2, 65, 3, 1, True), (ELASTICITY, 2, 54, 1, 1, False),
    (ELASTICITY, 2, 55, 1, 1, True), (ELASTICITY, 2, 64, 2, 1, False), (ELASTICITY, 2, 65, 2, 1, True),
    (ELASTICITY, 3, 9, 1, 1, False), (ELASTICITY, 3, 10, 1, 1, True), (ELASTICITY, 2, 40, 3, 4, False)])
def test_tuner_keeps_the_accurate_fp32_kernel_by_size(kind, dim, n, N, nrhs, simt):
    op = operator(kind, dim, n, N)
    for _ in range(3):
        entries = op.autotune(FP32, nrhs=nrhs)
        best = min(entries, key=lambda e: e["ms"])
        kept = op.apply_config(FP32)
        if simt:
            assert kept["family"] == "simt"
        else:
            assert kept == {k: best[k] for k in ("family", "ctas_per_sm", "tile")}


@pytest.mark.parametrize("kind,dim,n,N", [(POISSON, 2, 20, 1), (ELASTICITY, 2, 9, 2), (ELASTICITY, 3, 3, 1)])
@pytest.mark.parametrize("precision", [MIXED, TF32])
def test_mixed_precisions_run_face_centric_beside_the_simt_kernel(kind, dim, n, N, precision):
    """The same products as the face-centric configuration, added in FP64 in another order: 1e-12."""
    op = operator(kind, dim, n, N)
    x = torch.randn(op.ndof, dtype=torch.float64, device="cuda")
    y, ref = torch.empty_like(x), torch.empty_like(x)
    op.set_apply_config(FP32, "face")
    op.apply(x, ref, precision)
    op.set_apply_config(FP32, "simt")
    op.apply(x, y, precision)
    assert (y - ref).abs().max() <= 1e-12 * ref.abs().max()
