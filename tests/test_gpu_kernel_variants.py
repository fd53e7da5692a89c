"""The kernel a context runs: reading, setting and restoring the plain FP32
variant, and the same bits from every run of the same call."""
import numpy as np
import pytest

from baemm_b200 import _capi, meshes
from baemm_b200.helmholtz import APPLY_FP32, APPLY_FP64, APPLY_TC, Helmholtz_CUDA

from tests.helpers import crandn

pytestmark = pytest.mark.gpu


def _setup(grid, wc, wcs):
    coords, tris = meshes.torus(n_minor=grid[0], n_major=grid[1])
    kap = np.linspace(1.0, 6.0, wc // wcs)
    coeff = np.array([[0.3, -1j * k, 1.0, 0.4] for k in kap], np.complex128)
    blocks = [crandn(np.random.default_rng(s), coords.shape[0], wc) for s in (7, 8)]
    return coords, tris, blocks, (kap, coeff, wc, wcs)


def _apply(H, B, args):
    C = np.zeros_like(B)
    H.ApplyBoundaryOperators_PL(1.0, B, 0.0, C, *args)
    return C


@pytest.mark.parametrize("wc,wcs", [(16, 8), (32, 16)])
def test_restoring_the_variant_restores_the_kernel(wc, wcs):
    """A context whose variant was read, changed and set back runs what a new one runs."""
    coords, tris, (B, _), args = _setup((19, 54), wc, wcs)
    with Helmholtz_CUDA(coords, tris, meshes.fibonacci_sphere(4)) as H:
        first = _apply(H, B, args)
        for key in (_capi.TUNE_DENSE_VARIANT, _capi.TUNE_TC_SEGMENT, _capi.TUNE_TC_GEN_WARPS, _capi.TUNE_TC_CHUNKS,
                    _capi.TUNE_TC_STAGGER, _capi.TUNE_TC_CTAS, _capi.TUNE_TC_SHARE):
            H.SetTuning(key, H.GetTuning(key))
        assert np.array_equal(_apply(H, B, args), first)
        saved = H.GetKernelVariant()
        H.SetKernelVariant(1)
        _apply(H, B, args)
        H.SetKernelVariant(saved)
        assert H.GetKernelVariant() == saved
        assert np.array_equal(_apply(H, B, args), first)


@pytest.mark.parametrize("mode", [APPLY_FP32, APPLY_FP64, APPLY_TC])
@pytest.mark.parametrize("grid", [(15, 17), (19, 54), (41, 125)])
def test_same_bits_from_every_run(mode, grid):
    """510 triangles (one cluster of blocks per target block), 2052 (clusters and
    partial blocks) and 10250 (partial blocks, several waves): two runs of one
    context with another block in between, and a second context."""
    coords, tris, (B, other), args = _setup(grid, 32, 16)
    out = []
    for _ in range(2):
        with Helmholtz_CUDA(coords, tris, meshes.fibonacci_sphere(4)) as H:
            H.SetApplyMode(mode)
            for block in (B, other, B):
                C = _apply(H, block, args)
                if block is B:
                    out.append(C)
    for C in out[1:]:
        assert np.array_equal(C, out[0])
