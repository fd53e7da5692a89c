"""Kernels and dispatch rules at the sizes where they can go wrong: edges of
tiles, remainders, split and unsplit launches, against the FP64 oracle."""
import numpy as np
import pytest

from baemm_b200 import _capi, meshes
from baemm_b200.helmholtz import APPLY_FP32, APPLY_FP64, APPLY_TC, Helmholtz_CUDA
from oracle import oracle as O

from tests.helpers import crandn, relerr

pytestmark = pytest.mark.gpu

# The single-precision forms hold every operator to 1e-5 of the FP64 oracle
# (FP32 geometry of well-shaped triangles, two-level FP32 sums); the FP64 form
# to 1e-11.
TOL32, TOL64 = 1e-5, 1e-11
COEFF = {"bie": lambda k: [0.5, -1j * k, 1, 0], "dtn": lambda k: [0.5, -1j * k, 0, 1],
         "sl": lambda k: [0, 1j, 0, 0], "all": lambda k: [0.3 + 0.1j, 0.7 - 1j * k, 1 + 0.3j, 0.4 - 0.2j]}


def _apply(mode, grid, wc, wcs, cname, setup=lambda H: None):
    """(library, FP64 oracle) boundary applies on a torus of 2 * grid[0] * grid[1] triangles."""
    coords, tris = meshes.torus(n_minor=grid[0], n_major=grid[1])
    meas = meshes.fibonacci_sphere(4)
    kap = np.linspace(1.0, 6.0, wc // wcs)
    coeff = np.array([COEFF[cname](k) for k in kap], np.complex128)
    B = crandn(np.random.default_rng(7), coords.shape[0], wc)
    got, ref = np.zeros_like(B), np.zeros_like(B)
    with Helmholtz_CUDA(coords, tris, meas) as H:
        H.SetApplyMode(mode)
        setup(H)
        H.ApplyBoundaryOperators_PL(1.0, B, 0.0, got, kap, coeff, wc, wcs)
    O.Oracle(coords, tris, meas, precision=64).ApplyBoundaryOperators_PL(1.0, B, 0.0, ref, kap, coeff, wc, wcs)
    return got, ref


@pytest.mark.parametrize("ctas", [1, 5, 23, 148, 300])
def test_tensor_core_split_blocks(ctas):
    """Target blocks shared by one, a few and many CTAs (the sums of their workspace slots)."""
    got, ref = _apply(APPLY_TC, (13, 23), 64, 32, "bie", lambda H: H.SetTuning(_capi.TUNE_TC_CTAS, ctas))
    assert relerr(got, ref) < TOL32


@pytest.mark.parametrize("gen_warps,seg", [(16, 1), (16, 16), (8, 3)])
@pytest.mark.parametrize("grid", [(3, 3), (4, 4), (3, 8), (5, 13), (8, 8), (15, 17), (19, 54)])
@pytest.mark.parametrize("wc,wcs,cname", [(16, 16, "bie"), (32, 16, "all"), (32, 32, "dtn"), (64, 16, "bie"), (64, 32, "dtn"),
                                          (64, 64, "bie"), (64, 16, "all")])
def test_tensor_core_tiles(gen_warps, seg, grid, wc, wcs, cname):
    """18 to 2052 triangles: less than a 32-source tile, one half of it, whole
    tiles and remainders, with every number of groups per entry set and per unit."""
    def setup(H):
        H.SetTuning(_capi.TUNE_TC_GEN_WARPS, gen_warps)
        H.SetTuning(_capi.TUNE_TC_SEGMENT, seg)
    got, ref = _apply(APPLY_TC, grid, wc, wcs, cname, setup)
    assert relerr(got, ref) < TOL32


@pytest.mark.parametrize("variant", [None, 0, 1, 2])
@pytest.mark.parametrize("grid", [(3, 3), (4, 4), (5, 13), (16, 8), (15, 17), (16, 16), (19, 54)])
@pytest.mark.parametrize("wc,wcs,cname", [(16, 16, "bie"), (32, 32, "all"), (24, 8, "dtn"), (8, 4, "all"), (4, 2, "bie"),
                                          (3, 1, "sl")])
def test_plain_fp32_variants(variant, grid, wc, wcs, cname):
    """18 to 2052 triangles: less than a tile, whole tiles and one more, one and
    many source splits, blocks of targets that are full, partly filled and half
    empty, in every chunk size's kernel."""
    got, ref = _apply(APPLY_FP32, grid, wc, wcs, cname,
                      lambda H: variant is not None and H.SetKernelVariant(variant))
    assert relerr(got, ref) < TOL32


def test_kernel_variant_reads_back():
    coords, tris = meshes.icosphere(1)
    with Helmholtz_CUDA(coords, tris, meshes.fibonacci_sphere(4)) as H:
        assert H.GetKernelVariant() == 0
        for v in (2, 0, 1):
            H.SetKernelVariant(v)
            assert H.GetKernelVariant() == v


GRIDS64 = [(3, 3), (4, 4), (5, 13), (8, 8), (15, 17), (19, 54)]


@pytest.mark.parametrize("grid", GRIDS64)
@pytest.mark.parametrize("wc,wcs,cname", [(16, 16, "bie"), (32, 16, "all"), (48, 16, "dtn"), (32, 32, "sl"), (64, 64, "all"),
                                          (16, 8, "dtn"), (24, 8, "bie"), (8, 8, "all"), (8, 4, "all"), (2, 1, "sl")])
def test_fp64_units(grid, wc, wcs, cname):
    """18 to 2052 triangles (remainders of 8 sources and 16 targets, split and
    unsplit) in every work unit of the FP64 form and in the chunk sizes below 8."""
    got, ref = _apply(APPLY_FP64, grid, wc, wcs, cname)
    assert relerr(got, ref) < TOL64


def test_fp64_large_arguments():
    """Phases beyond the fast argument reduction: kappa r up to about 1e6.  A
    relative rounding of 1e-16 in r is 1e-10 in the phase there; 1e-8 leaves two digits."""
    coords, tris = meshes.torus(n_minor=5, n_major=13)
    B = crandn(np.random.default_rng(3), coords.shape[0], 16)
    got, ref = np.zeros_like(B), np.zeros_like(B)
    kap, coeff = np.array([2.0, 4e5]), np.array([COEFF["bie"](2.0), COEFF["all"](3.0)], np.complex128)
    with Helmholtz_CUDA(coords, tris, meshes.fibonacci_sphere(4)) as H:
        H.SetApplyMode(APPLY_FP64)
        H.ApplyBoundaryOperators_PL(1.0, B, 0.0, got, kap, coeff, 16, 8)
    O.Oracle(coords, tris, meshes.fibonacci_sphere(4), precision=64).ApplyBoundaryOperators_PL(
        1.0, B, 0.0, ref, kap, coeff, 16, 8)
    assert relerr(got, ref) < 1e-8


@pytest.mark.parametrize("count", [1, 15, 17, 64, 65, 300])
@pytest.mark.parametrize("wc,wcs", [(16, 16), (32, 16), (64, 32), (16, 8), (8, 8), (4, 2)])
def test_fp64_far_and_near(count, wc, wcs):
    """Directions and evaluation points that are not multiples of a block, beta on."""
    coords, tris = meshes.torus(n_minor=7, n_major=19)
    meas = meshes.fibonacci_sphere(count)
    points = meshes.points_off_torus(count, seed=5)
    kap = np.linspace(1.0, 5.0, wc // wcs)
    rng = np.random.default_rng(11)
    B, C0 = crandn(rng, coords.shape[0], wc), crandn(rng, count, wc)
    coeff = np.array([COEFF["all"](k) for k in kap], np.complex128)
    coeff[:, 3] = 0.0
    orc = O.Oracle(coords, tris, meas, precision=64)
    with Helmholtz_CUDA(coords, tris, meas) as H:
        H.SetApplyMode(APPLY_FP64)
        for name, extra in (("ApplyFarFieldOperators_PL", ()), ("ApplyNearFieldOperators_PL", (points,))):
            got, ref = C0.copy(), C0.copy()
            getattr(H, name)(0.7, B, 0.3, got, kap, coeff, wc, wcs, *extra)
            getattr(orc, name)(0.7, B, 0.3, ref, kap, coeff, wc, wcs, *extra)
            assert relerr(got, ref) < TOL64, name


def _bipyramid(n):
    """n equatorial vertices and two poles of degree n."""
    a = 2 * np.pi * np.arange(n) / n
    coords = np.concatenate([np.stack([np.cos(a), np.sin(a), 0 * a], 1), [[0, 0, 0.5], [0, 0, -0.5]]])
    i, j = np.arange(n), (np.arange(n) + 1) % n
    return coords, np.concatenate([np.stack([i, j, 0 * i + n], 1), np.stack([j, i, 0 * i + n + 1], 1)])


@pytest.mark.parametrize("ncols", [1, 5, 70])
@pytest.mark.parametrize("mesh", ["9", "511", "512", "513", "5125", "16384", "poles of degree 3", "poles of degree 60"])
def test_one_launch_mass_inverse(mesh, ncols):
    """Rows that do and do not fill the blocks of a cluster, matrix rows in and
    out of shared memory, and rows of the mass matrix with more than 8 entries."""
    grids = {"9": (3, 3), "511": (7, 73), "512": (16, 32), "513": (19, 27), "5125": (41, 125), "16384": (128, 128)}
    coords, tris = meshes.torus(n_minor=grids[mesh][0], n_major=grids[mesh][1]) if mesh in grids else \
        _bipyramid(int(mesh.split()[-1]))
    X = np.random.default_rng(ncols).standard_normal((coords.shape[0], ncols))
    got, ref = np.zeros_like(X), np.zeros_like(X)
    with Helmholtz_CUDA(coords, tris, np.eye(3)) as H:
        assert H.ProfileKrylov(1, 1, 1)["cg_iteration"]["one_launch_path"]
        for mode, tol in ((APPLY_FP64, TOL64), (APPLY_FP32, 1e-6)):   # FP32: mass values rounded to float
            H.SetApplyMode(mode)
            H.ApplyMassInverse(X, got, 1e-10)
            orc = O.Oracle(coords, tris, np.eye(3), precision=64 if mode == APPLY_FP64 else 32)
            for k in range(ncols):   # the oracle iterates a block until its last column has converged, the library each column
                one = np.zeros((coords.shape[0], 1))
                orc.ApplyMassInverse(np.ascontiguousarray(X[:, k:k + 1]), one, 1e-10)
                ref[:, k] = one[:, 0]
            assert relerr(got, ref) < tol, mode


def _mass_pattern(nv, tris):
    rows = [set() for _ in range(nv)]
    for t in np.asarray(tris).tolist():
        for v in t:
            rows[v].update(t)
    outer = np.concatenate([[0], np.cumsum([len(r) for r in rows])])
    return outer, np.concatenate([sorted(r) for r in rows if r]).astype(np.int32)


def _shuffled(mesh, extra=0):
    """The mesh with its triangles and vertices in random order, `extra` vertices in no triangle."""
    coords, tris = mesh
    rng = np.random.default_rng(1)
    perm = rng.permutation(len(coords) + extra)
    out = rng.standard_normal((len(coords) + extra, 3))
    out[perm[:len(coords)]] = coords
    return out, perm[np.asarray(tris)][rng.permutation(len(tris))]


@pytest.mark.parametrize("name,mesh", [
    ("one triangle", (np.eye(3), np.array([[2, 0, 1]]))), ("torus 3 x 3", meshes.torus(n_minor=3, n_major=3)),
    ("degree 64", _shuffled(_bipyramid(64), 3)), ("degree 65", _shuffled(_bipyramid(65), 3)),
    ("2046 vertices", _shuffled(meshes.torus(n_minor=31, n_major=66))),
    ("2047 vertices", _shuffled(meshes.torus(n_minor=23, n_major=89))),
    ("2048 vertices", _shuffled(meshes.torus(n_minor=32, n_major=64), 1)),
    ("icosphere 5", _shuffled(meshes.icosphere(5), 2))], ids=lambda p: p if isinstance(p, str) else "")
def test_topology(name, mesh):
    """Rows of the mass matrix (device and host construction, tiles of the scan)
    and an apply over the vertex -> triangle rows, re-meshing a context that held another mesh."""
    coords, tris = mesh
    with Helmholtz_CUDA(*meshes.icosphere(2), np.eye(3)) as H:
        H.SetMesh(coords, tris)
        outer, inner, vals = H.MassMatrix()
        ref_outer, ref_inner = _mass_pattern(len(coords), tris)
        assert np.array_equal(outer, ref_outer) and np.array_equal(inner, ref_inner)
        p = coords[tris]
        area = 0.5 * np.linalg.norm(np.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]), axis=1)
        assert abs(vals.sum() - area.sum()) < 1e-5 * area.sum()
        if name in ("icosphere 5", "degree 65"):
            X = np.random.default_rng(2).standard_normal((len(coords), 2))
            got, ref = np.zeros_like(X), np.zeros_like(X)
            w = area[:, None, None] / 12
            np.add.at(ref, tris, w * (X[tris] + X[tris].sum(axis=1, keepdims=True)))
            assert relerr(H.MassDot(1.0, X, 0.0, got), ref) < TOL32
            kap, coeff = np.array([2.0]), np.array([COEFF["bie"](2.0)], np.complex128)
            B = crandn(np.random.default_rng(3), len(coords), 4)
            got, ref = np.zeros_like(B), np.zeros_like(B)
            H.SetApplyMode(APPLY_FP64)
            H.ApplyBoundaryOperators_PL(1.0, B, 0.0, got, kap, coeff, 4, 4)
            O.Oracle(coords, tris, np.eye(3), precision=64).ApplyBoundaryOperators_PL(1.0, B, 0.0, ref, kap, coeff, 4, 4)
            used = np.unique(tris)
            assert relerr(got[used], ref[used]) < TOL64


@pytest.mark.parametrize("grid", [(3, 3), (7, 73), (16, 32), (41, 125)])
@pytest.mark.parametrize("chunks,directions", [(1, 1), (1, 2), (2, 16), (1, 64)])
def test_one_launch_arnoldi(grid, chunks, directions):
    """A solve to 1e-10 and its residual by the FP64 apply: 1 to 64 columns (half a
    pair, one, many), rows that do and do not fill the blocks of a cluster.
    The solve ends on |P r| <= 1e-10 |P b|; the residual itself is held to 1e-8
    (the condition of the mass matrix, below 100 on these grids)."""
    coords, tris = meshes.torus(n_minor=grid[0], n_major=grid[1])
    kap = np.array([1.0, 2.0][:chunks])
    wave = crandn(np.random.default_rng(5), coords.shape[0], chunks * directions)
    phi, back = np.zeros_like(wave), np.zeros_like(wave)
    coeff = np.zeros((chunks, 4), np.complex128)
    with Helmholtz_CUDA(coords, tris, np.eye(3)) as H:
        H.SetApplyMode(APPLY_FP64)
        H.BoundaryPotential(kap, coeff, wave, phi, directions, 1e-12, 1e-10)
        assert H.LastSolveStats()["gmres_converged"]
        H.ApplyBoundaryOperators_PL(1.0, phi, 0.0, back, kap, coeff, wave.shape[1], directions)
    assert relerr(back, wave) < 1e-8


@pytest.mark.parametrize("wc", [16, 416, 448])
@pytest.mark.parametrize("mode,tol", [(APPLY_FP32, TOL32), (APPLY_FP64, TOL64)])
def test_averaging_of_few_and_many_rows(mode, tol, wc):
    """512 vertices in launches of 512, 6656 and 7168 warps: below and above three
    quarters of what the chip holds, where the row loops of the epilogue change."""
    got, ref = _apply(mode, (16, 32), wc, 16, "all")
    assert relerr(got, ref) < tol


@pytest.mark.parametrize("mode,tol", [(APPLY_FP32, TOL32), (APPLY_FP64, TOL64)])
def test_split_launch_under_capture(mode, tol):
    """A caller captures an apply of 16 columns in a context that has only run 256:
    the narrow launch is split over the sources, the wide one was not, and under
    capture the partial blocks have to make do with the room there is.  The same
    for the far field."""
    import torch
    coords, tris = meshes.torus(n_minor=32, n_major=80)
    s = torch.cuda.Stream()
    B = torch.as_tensor(crandn(np.random.default_rng(3), coords.shape[0], 256)).cuda()
    C, narrow = torch.zeros_like(B), B[:, :16].contiguous()
    Cn, again = torch.zeros_like(narrow), torch.zeros_like(narrow)
    meas = meshes.fibonacci_sphere(70)
    B2, n2 = B.to(torch.complex128), narrow.to(torch.complex128)
    F, Fn = B2.new_zeros(70, 256), B2.new_zeros(70, 16)
    coeff = lambda ks: np.array([COEFF["bie"](k) for k in ks], np.complex128)
    with Helmholtz_CUDA(coords, tris, meas) as H:
        H.SetApplyMode(mode)
        H.SetStream(s.cuda_stream)
        torch.cuda.synchronize()
        wide = np.linspace(1.0, 6.0, 16)
        H.ApplyBoundaryOperators_PL(1.0, B, 0.0, C, wide, coeff(wide), 256, 16)
        H.ApplyFarFieldOperators_PL(1.0, B2, 0.0, F, wide, coeff(wide), 256, 16)
        H.LoadBoundaryOperators_PL(np.array([2.0]), coeff([2.0]), 16, 16)
        H.Synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            H.ApplyBoundaryOperators_PL(1.0, narrow, 0.0, Cn)
            H.ApplyFarFieldOperators_PL(1.0, n2, 0.0, Fn)
        g.replay()
        H.ApplyBoundaryOperators_PL(1.0, narrow, 0.0, again)
        torch.cuda.synchronize()
        H.UnloadBoundaryOperators_PL()
        H.SetStream(None)
        del g
    ref, fref = np.zeros((coords.shape[0], 16), np.complex128), np.zeros((70, 16), np.complex128)
    orc, args = O.Oracle(coords, tris, meas, precision=64), (np.array([2.0]), coeff([2.0]), 16, 16)
    orc.ApplyBoundaryOperators_PL(1.0, narrow.cpu().numpy(), 0.0, ref, *args)
    orc.ApplyFarFieldOperators_PL(1.0, n2.cpu().numpy(), 0.0, fref, *args)
    assert relerr(Fn.cpu().numpy(), fref) < tol
    assert relerr(Cn.cpu().numpy(), ref) < tol
    assert relerr(again.cpu().numpy(), ref) < tol
