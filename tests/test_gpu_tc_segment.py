"""The tensor-core form's segment setting bounds the accumulation chain: never
more groups of 16 sources than asked for, a single one included."""
import numpy as np
import pytest

from baemm_b200 import _capi, meshes
from baemm_b200.helmholtz import APPLY_TC, Helmholtz_CUDA
from oracle import oracle as O

from tests.helpers import crandn, relerr

pytestmark = pytest.mark.gpu

TOL = 1e-5   # the bar of the single-precision forms against the FP64 oracle


def _setup(grid, wc, wcs, cname="bie"):
    coords, tris = meshes.torus(n_minor=grid[0], n_major=grid[1])
    kap = np.linspace(1.0, 6.0, wc // wcs)
    coeff = np.array([[0.3, -1j * k, 1.0, 0.0] if cname == "bie" else [0.3 + 0.1j, 0.7 - 1j * k, 1 + 0.3j, 0.4 - 0.2j]
                      for k in kap], np.complex128)
    return coords, tris, crandn(np.random.default_rng(7), coords.shape[0], wc), (kap, coeff, wc, wcs)


@pytest.mark.parametrize("gen_warps", [16, 8])
@pytest.mark.parametrize("grid", [(3, 3), (4, 4), (3, 8), (5, 13), (8, 8), (19, 54)])
@pytest.mark.parametrize("wc,wcs,cname", [(16, 16, "bie"), (64, 16, "all"), (64, 32, "bie"), (64, 64, "bie")])
def test_single_group(gen_warps, grid, wc, wcs, cname):
    """Tiles of 16 sources (18 to 2052 triangles): boundary, row shards that cut
    through a tile, and the near field, in another order of summation than tiles of 32."""
    coords, tris, B, args = _setup(grid, wc, wcs, cname)
    kap, coeff, _, _ = args
    points = meshes.points_off_torus(77, seed=5)
    near = coeff.copy()
    near[:, 0] = near[:, 3] = 0
    out = {}
    with Helmholtz_CUDA(coords, tris, np.eye(3)) as H:
        H.SetApplyMode(APPLY_TC)
        H.SetTuning(_capi.TUNE_TC_GEN_WARPS, gen_warps)
        for seg in (1, 2, 1):
            H.SetTuning(_capi.TUNE_TC_SEGMENT, seg)
            C, F = np.zeros_like(B), np.zeros((77, wc), complex)
            H.ApplyBoundaryOperators_PL(1.0, B, 0.0, C, *args)
            H.ApplyNearFieldOperators_PL(1.0, B, 0.0, F, kap, near, wc, wcs, points)
            if seg in out:
                assert np.array_equal(C, out[seg][0]) and np.array_equal(F, out[seg][1])
            out[seg] = C, F
        import torch
        Bd = torch.from_numpy(B).cuda()
        H.LoadBoundaryOperators_PL(*args)
        shards = torch.zeros_like(Bd)
        n, cut = tris.shape[0], tris.shape[0] // 2 + 1
        for k, (a, b) in enumerate(((0, cut), (cut, n))):
            P = torch.zeros_like(Bd)
            H.ApplyBoundaryOperatorsRows(1.0, Bd, 0.0, P, a, b, with_mass=(k == 0))
            shards += P
        shards = shards.cpu().numpy()
        H.UnloadBoundaryOperators_PL()
    orc = O.Oracle(coords, tris, np.eye(3), precision=64)
    ref, fref = np.zeros_like(B), np.zeros((77, wc), complex)
    orc.ApplyBoundaryOperators_PL(1.0, B, 0.0, ref, *args)
    orc.ApplyNearFieldOperators_PL(1.0, B, 0.0, fref, kap, near, wc, wcs, points)
    assert relerr(out[1][0], ref) < TOL and relerr(out[1][1], fref) < TOL and relerr(shards, ref) < TOL
    if tris.shape[0] > 16:   # more than one segment
        assert not np.array_equal(out[1][0], out[2][0])


def test_odd_settings_accumulate_no_more_than_asked():
    coords, tris, B, args = _setup((19, 54), 32, 16)
    out = {}
    with Helmholtz_CUDA(coords, tris, np.eye(3)) as H:
        H.SetApplyMode(APPLY_TC)
        for seg in (2, 3, 4, 5, 6):
            H.SetTuning(_capi.TUNE_TC_SEGMENT, seg)
            assert H.GetTuning(_capi.TUNE_TC_SEGMENT) == seg
            out[seg] = np.zeros_like(B)
            H.ApplyBoundaryOperators_PL(1.0, B, 0.0, out[seg], *args)
    assert np.array_equal(out[3], out[2]) and np.array_equal(out[5], out[4])
    assert not np.array_equal(out[4], out[2]) and not np.array_equal(out[6], out[4])


def test_single_group_in_packed_launches():
    """A solve whose dense stage runs in a packer's launches, with the same setting."""
    from baemm_b200 import Packer
    coords, tris = meshes.icosphere(3)
    wave = crandn(np.random.default_rng(3), coords.shape[0], 16)
    phi = []
    for packed in (False, True):
        with Packer(0, max_wait_us=1000) as P, Helmholtz_CUDA(coords, tris, np.eye(3)) as H:
            H.SetApplyMode(APPLY_TC)
            H.SetTuning(_capi.TUNE_TC_SEGMENT, 1)
            if packed:
                H.SetPacker(P)
            phi.append(np.zeros_like(wave))
            H.BoundaryPotential(np.array([3.0]), np.zeros((1, 4), complex), wave, phi[-1], 16, 1e-10, 1e-6)
            assert H.LastSolveStats()["gmres_converged"]
            if packed:
                assert P.stats()["launches"] > 0
                H.SetPacker(None)
    assert relerr(phi[1], phi[0]) < TOL
