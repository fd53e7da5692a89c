"""Work buffers over the life of a context: a call on a mesh, columns and points
no larger than earlier ones' allocates nothing, so what a caller captured in a
CUDA graph of its own stays valid."""
import numpy as np
import pytest

from baemm_b200 import meshes
from baemm_b200.helmholtz import APPLY_FP32, APPLY_FP64, APPLY_TC, Helmholtz_CUDA

from tests.helpers import crandn, relerr

pytestmark = pytest.mark.gpu

MEAS = meshes.fibonacci_sphere(70)
LARGE = (50, 128)   # 12800 triangles; 256 columns fill the chip without a split over the sources, fewer do not
# (grid, columns, evaluation points) of calls no larger than LARGE, 256 columns, 4000 points
SMALLER = [(LARGE, 96, 4000), (LARGE, 16, 333), (LARGE, 64, 1000), ((32, 80), 64, 4000), ((32, 80), 16, 1000),
           ((20, 64), 256, 4000), ((4, 4), 256, 64)]


def _mesh(grid):
    return meshes.torus(n_minor=grid[0], n_major=grid[1])


def _calls(H, coords, wc, points):
    """A boundary, a near-field and a far-field apply of host blocks."""
    kap = np.linspace(1.0, 5.0, wc // 16)
    coeff = np.array([[0.5, -1j * k, 1.0, 0.0] for k in kap])
    B = crandn(np.random.default_rng(wc), coords.shape[0], wc)
    out = [np.zeros_like(B), np.zeros((points, wc), complex), np.zeros((70, wc), complex)]
    H.ApplyBoundaryOperators_PL(1.0, B, 0.0, out[0], kap, coeff, wc, 16)
    coeff[:, 0] = 0.0
    H.ApplyNearFieldOperators_PL(1.0, B, 0.0, out[1], kap, coeff, wc, 16, meshes.points_off_torus(points, seed=5))
    H.ApplyFarFieldOperators_PL(1.0, B, 0.0, out[2], kap, coeff, wc, 16)
    return out


@pytest.mark.parametrize("mode", [APPLY_FP32, APPLY_FP64, APPLY_TC])
def test_smaller_calls_allocate_nothing(mode):
    import torch
    alone = []
    for grid, wc, points in SMALLER:   # in contexts of their own (and every kernel is loaded)
        coords, tris = _mesh(grid)
        with Helmholtz_CUDA(coords, tris, MEAS) as H:
            H.SetApplyMode(mode)
            alone.append(_calls(H, coords, wc, points))
    coords, tris = _mesh(LARGE)
    with Helmholtz_CUDA(coords, tris, MEAS) as H:
        H.SetApplyMode(mode)
        _calls(H, coords, 256, 4000)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        for (grid, wc, points), ref in zip(SMALLER, alone):
            coords, tris = _mesh(grid)
            H.SetMesh(coords, tris)
            for a, b in zip(_calls(H, coords, wc, points), ref):
                assert np.array_equal(a, b), (grid, wc)
            assert torch.cuda.mem_get_info()[0] == free, (grid, wc)


@pytest.mark.parametrize("mode", [APPLY_FP32, APPLY_FP64])
def test_captured_applies_survive_smaller_calls(mode):
    """A caller's graph of a split boundary and a split far-field apply, replayed
    after other applies of the context, none larger, have run."""
    import torch
    coords, tris = _mesh(LARGE)
    s = torch.cuda.Stream()
    kap = np.array([1.0, 4.0])
    coeff = np.array([[0.5, -1j * k, 1.0, 0.0] for k in kap])
    B = torch.as_tensor(crandn(np.random.default_rng(3), coords.shape[0], 32)).cuda()
    C, F = torch.zeros_like(B), B.new_zeros(70, 32)
    with Helmholtz_CUDA(coords, tris, MEAS) as H:
        H.SetApplyMode(mode)
        H.SetStream(s.cuda_stream)
        H.LoadBoundaryOperators_PL(kap, coeff, 32, 16)
        torch.cuda.synchronize()

        def applies():
            H.ApplyBoundaryOperators_PL(1.0, B, 0.0, C)
            H.ApplyFarFieldOperators_PL(1.0, B, 0.0, F)
        applies()
        torch.cuda.synchronize()
        ref = C.clone(), F.clone()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            applies()
        for rows in ((0, 1000), (3000, 3500), (100, 12000)):   # shards: other splits of the same operators
            H.ApplyBoundaryOperatorsRows(1.0, B, 0.0, torch.zeros_like(B), *rows)
        H.LoadBoundaryOperators_PL(kap[:1], coeff[:1], 16, 16)
        for op, rows in ((H.ApplyBoundaryOperators_PL, coords.shape[0]), (H.ApplyFarFieldOperators_PL, 70)):
            op(1.0, B[:, :16].contiguous(), 0.0, B.new_zeros(rows, 16))
        torch.cuda.synchronize()
        H.LoadBoundaryOperators_PL(kap, coeff, 32, 16)   # the graph reads the loaded parameters
        C.zero_()
        F.zero_()
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(C, ref[0]) and torch.equal(F, ref[1])
        del g
        H.UnloadBoundaryOperators_PL()
        H.SetStream(None)


def test_capture_without_room_for_a_split():
    """The tensor-core form leaves no partial blocks; a capture of the plain form
    after it must not allocate them."""
    import torch
    coords, tris = _mesh((32, 80))
    s = torch.cuda.Stream()
    kap, coeff = np.array([2.0]), np.array([[0.5, -2j, 1.0, 0.0]])
    B = torch.as_tensor(crandn(np.random.default_rng(3), coords.shape[0], 16)).cuda().to(torch.complex64)
    C, split = torch.zeros_like(B), torch.zeros_like(B)
    with Helmholtz_CUDA(coords, tris, MEAS) as H:   # loads the kernels, and the split form's values
        H.ApplyBoundaryOperators_PL(1.0, B, 0.0, split, kap, coeff, 16, 16)
        torch.cuda.synchronize()
    with Helmholtz_CUDA(coords, tris, MEAS) as H:
        H.SetStream(s.cuda_stream)
        H.SetApplyMode(APPLY_TC)
        H.LoadBoundaryOperators_PL(kap, coeff, 16, 16)
        torch.cuda.synchronize()
        H.ApplyBoundaryOperators_PL(1.0, B, 0.0, C)
        torch.cuda.synchronize()
        H.SetApplyMode(APPLY_FP32)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            H.ApplyBoundaryOperators_PL(1.0, B, 0.0, C)
        g.replay()
        torch.cuda.synchronize()
        assert not torch.equal(C, split)   # one sum over all sources, in another order
        assert relerr(C.cpu().numpy(), split.cpu().numpy()) < 1e-5
        del g
        H.UnloadBoundaryOperators_PL()
        H.SetStream(None)


@pytest.mark.parametrize("mode,tol", [(APPLY_FP32, 1e-5), (APPLY_FP64, 1e-11)])
def test_capture_in_the_room_of_another_shape(mode, tol):
    """512 triangles x 256 columns leave work blocks as large as 8192 x 16 needs, no
    partial blocks and fewer of the far field's than that would take: captured, the
    larger mesh makes do with the room there is and allocates nothing."""
    import torch
    coords, tris = _mesh((64, 64))
    s = torch.cuda.Stream()
    kap, coeff = np.array([2.0]), np.array([[0.5, -2j, 1.0, 0.0]])
    B = torch.as_tensor(crandn(np.random.default_rng(3), coords.shape[0], 16)).cuda()
    C, F, free_c, free_f = (torch.zeros_like(B), B.new_zeros(70, 16), torch.zeros_like(B), B.new_zeros(70, 16))
    with Helmholtz_CUDA(coords, tris, MEAS) as H:   # with all the room it takes
        H.SetApplyMode(mode)
        H.LoadBoundaryOperators_PL(kap, coeff, 16, 16)
        H.ApplyBoundaryOperators_PL(1.0, B, 0.0, free_c)
        H.ApplyFarFieldOperators_PL(1.0, B, 0.0, free_f)
        torch.cuda.synchronize()
    small = _mesh((16, 16))
    with Helmholtz_CUDA(*small, MEAS) as H:
        H.SetApplyMode(mode)
        wide = np.linspace(1.0, 5.0, 16)
        wide_coeff = np.array([[0.5, -1j * k, 1.0, 0.0] for k in wide])
        W = np.ones((256, 256), complex)
        H.ApplyBoundaryOperators_PL(1.0, W, 0.0, np.zeros_like(W), wide, wide_coeff, 256, 16)
        H.ApplyFarFieldOperators_PL(1.0, W, 0.0, np.zeros((70, 256), complex), wide, wide_coeff, 256, 16)
        H.SetMesh(coords, tris)
        H.SetStream(s.cuda_stream)
        H.LoadBoundaryOperators_PL(kap, coeff, 16, 16)
        H.Synchronize()
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            before = torch.cuda.mem_get_info()[0]
            H.ApplyBoundaryOperators_PL(1.0, B, 0.0, C)
            H.ApplyFarFieldOperators_PL(1.0, B, 0.0, F)
            assert torch.cuda.mem_get_info()[0] == before
        g.replay()
        torch.cuda.synchronize()
        for a, b in ((C, free_c), (F, free_f)):
            assert relerr(a.cpu().numpy(), b.cpu().numpy()) < tol
        assert not torch.equal(C, free_c)   # split less: in another order
        if mode == APPLY_FP64:   # in FP32 both far fields have the parts they would choose
            assert not torch.equal(F, free_f)
        del g
        H.UnloadBoundaryOperators_PL()
        H.SetStream(None)
