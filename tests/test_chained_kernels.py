"""Kernels that start while the one in front of them finishes (launch_chained).

What an earlier kernel of the chain writes is not read-only while a chained
kernel lives, so it must not be read through the read-only path: the sources
are checked on the CPU, and applies that follow one another without a wait of
the host are compared with the same applies each run alone on the GPU."""
import glob
import os
import re

import numpy as np
import pytest

from baemm_b200 import meshes
from baemm_b200.helmholtz import APPLY_FP32, APPLY_FP64, APPLY_TC, Helmholtz_CUDA

from tests.helpers import crandn

CSRC = os.path.join(os.path.dirname(__file__), "..", "baemm_b200", "csrc")
# read by chained kernels and written by none: the mesh, its matrices, the parameters of the operators
CONSTANT = {"tri_sorted", "a3", "avt_outer", "avt_inner", "diag", "prm", "m_outer", "m_inner", "m_val", "mid4", "nrm4",
            "mo", "mi", "mv", "ell_idx", "ell_val", "L", "tgeo"}


def _chained():
    """(kernel, its parameter list, its body) of every kernel that launch_chained launches."""
    text = {f: open(f).read() for f in sorted(glob.glob(os.path.join(CSRC, "*.cu")))}
    names = {n for t in text.values() for n in re.findall(r"launch_chained\((?:few \? )?(\w+)", t)}
    for name in sorted(names):
        for t in text.values():
            m = re.search(r"\b%s\(([^;{]*)\)\s*\n\{(.*?)\n\}\n" % name, t, re.S)
            if m:
                yield name, m.group(1), m.group(2)
                break
        else:
            raise AssertionError(f"no definition of {name} found")


def test_chained_kernels_read_what_the_chain_writes_through_plain_pointers():
    kernels = list(_chained())
    assert len(kernels) >= 12
    for name, params, body in kernels:
        assert re.search(r"\bchain_(wait|begin)\(\)", body), f"{name} does not wait for the kernel in front of it"
        restricted = set(re.findall(r"const[^,]*?__restrict__\s+(\w+)", params))
        assert restricted <= CONSTANT, f"{name}: {restricted - CONSTANT} may be read before the wait"
    # the Arnoldi step reads vectors that the host has waited for before the launch
    arnoldi = next(body for name, _, body in kernels if name == "arnoldi_kernel")
    assert set(re.findall(r"\b__ldg\((.*?)\)", arnoldi)) <= {"p + i * stride"}
    for f in glob.glob(os.path.join(CSRC, "*.cu")):
        assert not re.search(r"\b__ldg\(", open(f).read().replace(arnoldi, "")), f


@pytest.mark.gpu
@pytest.mark.parametrize("mode,wc,wcs", [(APPLY_FP32, 16, 8), (APPLY_TC, 32, 16), (APPLY_FP64, 16, 16)])
@pytest.mark.parametrize("grid", [(4, 9), (15, 17), (32, 80)])
def test_applies_without_a_wait_between_them(mode, wc, wcs, grid):
    """Boundary, near- and far-field applies of changing blocks into the same work
    buffers, enqueued back to back: bit for bit what each gives alone."""
    import torch
    coords, tris = meshes.torus(n_minor=grid[0], n_major=grid[1])
    rng = np.random.default_rng(3)
    kap = np.linspace(1.0, 5.0, wc // wcs)
    coeff = np.array([[0.5, -1j * k, 1.0, 0.0] for k in kap])
    coeff_near = np.array([[0.0, -1j * k, 1.0, 0.0] for k in kap])
    real = torch.complex128 if mode == APPLY_FP64 else torch.complex64
    meas = meshes.fibonacci_sphere(70)
    points = torch.from_numpy(meshes.points_off_torus(333, seed=5)).cuda()
    blocks = [torch.from_numpy(crandn(rng, coords.shape[0], wc)).cuda().to(real) for _ in range(8)]
    stream = torch.cuda.Stream()
    with Helmholtz_CUDA(coords, tris, meas) as H:
        H.SetApplyMode(mode)
        H.SetStream(stream.cuda_stream)   # one stream throughout: nothing is recorded between the applies

        def passes(wait):
            out = []
            for what in ("ApplyBoundaryOperators_PL", "ApplyNearFieldOperators_PL", "ApplyFarFieldOperators_PL"):
                H.LoadBoundaryOperators_PL(kap, coeff if what == "ApplyBoundaryOperators_PL" else coeff_near, wc, wcs)
                far = what == "ApplyFarFieldOperators_PL"
                ins = [b.to(torch.complex128) if far else b for b in blocks]
                rows = 70 if far else 333 if "Near" in what else coords.shape[0]
                res = [torch.zeros(rows, wc, dtype=x.dtype, device="cuda") for x in ins]
                extra = (points,) if "Near" in what else ()
                torch.cuda.synchronize()
                for x, y in zip(ins, res):
                    getattr(H, what)(1.0, x, 0.0, y, *extra)
                    if wait:
                        torch.cuda.synchronize()
                torch.cuda.synchronize()
                H.UnloadBoundaryOperators_PL()
                out += [y.cpu() for y in res]
            return out

        alone = passes(True)
        for _ in range(3):
            for a, b in zip(alone, passes(False)):
                assert torch.equal(a, b)
        H.SetStream(None)
