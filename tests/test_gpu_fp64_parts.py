"""The FP64 form keeps the accuracy of the real and of the imaginary part, each
by itself: low frequencies (imaginary parts of the kernel far below the real
ones), blocks whose parts differ by many orders."""
import numpy as np
import pytest

from baemm_b200 import meshes
from baemm_b200.helmholtz import APPLY_FP64, Helmholtz_CUDA
from oracle import oracle as O

from tests.helpers import relerr

pytestmark = pytest.mark.gpu

# Sums of at most 2048 terms of one sign, every term within a few units of 2^-53 of
# its own value: 2048 * 2^-53 = 2.3e-13 at the very most.
TOL = 1e-12
KAPPA = 1e-8   # the imaginary parts are about 1e-8 of the real ones


def _run(coeff, B, name="ApplyBoundaryOperators_PL", wcs=16, kappa=KAPPA):
    """(library, oracle) of one operator on a torus of 510 triangles."""
    coords, tris = meshes.torus(n_minor=15, n_major=17)
    meas = meshes.fibonacci_sphere(33)
    wc = B.shape[1]
    args = (np.full(wc // wcs, kappa), np.tile(np.array(coeff, np.complex128), (wc // wcs, 1)), wc, wcs)
    if "Near" in name:
        args += (3.0 * meshes.fibonacci_sphere(33),)
    rows = coords.shape[0] if "Boundary" in name else 33
    got, ref = np.zeros((rows, wc), complex), np.zeros((rows, wc), complex)
    with Helmholtz_CUDA(coords, tris, meas) as H:
        H.SetApplyMode(APPLY_FP64)
        getattr(H, name)(1.0, B, 0.0, got, *args)
    getattr(O.Oracle(coords, tris, meas, precision=64), name)(1.0, B, 0.0, ref, *args)
    return got, ref


@pytest.mark.parametrize("wc,wcs", [(16, 16), (32, 16), (32, 32), (8, 8), (4, 2)])
@pytest.mark.parametrize("name", ["ApplyBoundaryOperators_PL", "ApplyNearFieldOperators_PL"])
def test_low_frequency_single_layer(name, wc, wcs):
    """c1 = 1 on a positive real density: Im A = kappa to first order."""
    B = np.random.default_rng(1).uniform(0.5, 1.5, (255, wc)).astype(complex)
    got, ref = _run([0, 1, 0, 0], B, name, wcs)
    assert relerr(got.real, ref.real) < TOL
    assert relerr(got.imag, ref.imag) < TOL


@pytest.mark.parametrize("name", ["ApplyBoundaryOperators_PL", "ApplyNearFieldOperators_PL", "ApplyFarFieldOperators_PL"])
def test_block_with_a_small_part(name):
    """kappa = 0: a real operator applies to both parts alike, however small one is."""
    rng = np.random.default_rng(2)
    B = rng.uniform(0.5, 1.5, (255, 16)) + 1e-9j * rng.uniform(0.5, 1.5, (255, 16))
    got, ref = _run([0, 1, 0, 0], B, name, kappa=0.0)
    assert relerr(got.real, ref.real) < TOL
    assert relerr(got.imag, ref.imag) < TOL


@pytest.mark.parametrize("name,coeff", [
    ("ApplyBoundaryOperators_PL", [0, 1e-60 + 1j, 0, 0]), ("ApplyBoundaryOperators_PL", [0, 0, 1 + 1e-60j, 0]),
    ("ApplyBoundaryOperators_PL", [0, 0, 0, 1 + 1e-60j]), ("ApplyNearFieldOperators_PL", [0, 1e-60 + 1j, 0, 0]),
    ("ApplyNearFieldOperators_PL", [0, 0, 1 + 1e-60j, 0])])
def test_coefficient_parts_below_single_precision(name, coeff):
    """kappa = 0 on a real block: one part of the result is the tiny part of the
    coefficient times what the other part is the large one times."""
    B = np.random.default_rng(4).uniform(0.5, 1.5, (255, 16)).astype(complex)
    got, ref = _run(coeff, B, name, kappa=0.0)
    small, large = (got.real, got.imag) if coeff[1] else (got.imag, got.real)
    assert np.abs(large).max() > 0
    assert relerr(small * 1e60, large) < TOL
    assert relerr(got, ref) < TOL
