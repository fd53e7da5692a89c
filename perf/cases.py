"""The work that programs have this library do, as cases to measure.

A case is a dict of plain values.  Kinds:

  apply    one boundary-operator apply on a block of right-hand sides: the step
           that every Krylov iteration repeats.  `op` is the operator of a solve:
           "bie" (1/2 M - i kappa SL + DL, the mixed boundary integral equation),
           "dtn" (1/2 M - i kappa SL + DL', its adjoint, the Dirichlet-to-Neumann
           solve of the derivatives) or "all" (every layer, complex coefficients).
  near     the boundary potential at points off the surface.
  far      the far field of a density in FP64.
  request  one request of a serving slot: a new mesh into a live context, then the
           scattering solve to its far field.
  adjoint  the adjoint shape derivative of the far field (the backward direction
           of a Gauss-Newton step): one refined solve with its waves and projections.

`mode` is the arithmetic ("fp32" is what a context does by default, "tc" the
compensated tensor-core form, "fp64"); blocks are complex64, in FP64 complex128.
`mesh` is "torus" (a x b grid, 2 a b triangles: any size, any remainder) or "sphere"
(an icosphere of level a, its radius perturbed as a shape iterate's is).
`chunks` wavenumbers (not more than 4) share the columns in chunks of `chunk_size`.
"""
import math

import numpy as np
import torch

from baemm_b200.helmholtz import APPLY_FP32, APPLY_FP64, APPLY_TC, Helmholtz_CUDA, WaveType
from baemm_b200.meshes import fibonacci_sphere, points_off_torus, sh_perturbed_sphere, torus

MODES = {"fp32": APPLY_FP32, "tc": APPLY_TC, "fp64": APPLY_FP64}
WAVENUMBERS = {1: [8.0], 2: [4.0, 8.0], 4: [2.0, 4.0, 8.0, 16.0]}
GMRES_TOL, CG_TOL, INNER_TOL, REFINEMENTS = 1e-10, 1e-10, 1e-6, 10


def listed():
    return [
        # latency: a coarse mesh, one wavenumber; what a first experiment or a unit test runs
        dict(name="apply-fp32-smallest", kind="apply", mode="fp32", op="bie", mesh="sphere", a=2, b=0,
             chunks=1, chunk_size=16, host=False),
        # the drop-in caller: host arrays, parameters with every call, eight directions (not a 16-column chunk)
        dict(name="apply-fp32-host", kind="apply", mode="fp32", op="bie", mesh="sphere", a=4, b=0,
             chunks=2, chunk_size=8, host=True),
        # the default arithmetic on an ordinary ragged mesh, the adjoint operator of the derivative solves
        dict(name="apply-fp32-dtn", kind="apply", mode="fp32", op="dtn", mesh="torus", a=67, b=151,
             chunks=2, chunk_size=16, host=False),
        # one apply inside a served request: one wavenumber, 32 waves, a small mesh
        dict(name="apply-tc-serving", kind="apply", mode="tc", op="bie", mesh="sphere", a=4, b=0,
             chunks=1, chunk_size=32, host=False),
        # one apply inside a Gauss-Newton step: two wavenumbers x 32 waves
        dict(name="apply-tc-gauss-newton", kind="apply", mode="tc", op="dtn", mesh="sphere", a=5, b=0,
             chunks=2, chunk_size=32, host=False),
        # the headline: 153,600 triangles, 64 right-hand sides over four wavenumbers
        dict(name="apply-tc-torus", kind="apply", mode="tc", op="bie", mesh="torus", a=160, b=480,
             chunks=4, chunk_size=16, host=False),
        # FP64 reference solves and the residuals of iterative refinement, small and ordinary
        dict(name="apply-fp64-small", kind="apply", mode="fp64", op="bie", mesh="sphere", a=3, b=0,
             chunks=2, chunk_size=16, host=False),
        dict(name="apply-fp64-ordinary", kind="apply", mode="fp64", op="bie", mesh="torus", a=83, b=251,
             chunks=2, chunk_size=16, host=False),
        # the scattered wave at points around the object (a field plot): ragged in points and triangles
        dict(name="near-tc", kind="near", mode="tc", op="bie", mesh="torus", a=71, b=213,
             chunks=2, chunk_size=16, points=20011),
        # the far-field map of a refined solve
        dict(name="far-fp64", kind="far", mode="fp64", op="bie", mesh="sphere", a=6, b=0,
             chunks=2, chunk_size=16, directions=256),
        # a served request to full accuracy: re-mesh, then the tensor-core solve inside FP64 refinement
        dict(name="request-refined", kind="request", mode="tc", op="bie", mesh="sphere", a=4, b=0,
             chunks=1, chunk_size=32, directions=128),
        # the backward half of a shape-optimisation step
        dict(name="adjoint-refined", kind="adjoint", mode="tc", op="dtn", mesh="sphere", a=5, b=0,
             chunks=2, chunk_size=16, directions=200),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["apply"] * 5 + ["near", "far", "request", "adjoint"])
    chunks = rng.choice([1, 2, 4])
    if kind in ("request", "adjoint"):
        case = dict(kind=kind, mode="tc", op="bie" if kind == "request" else "dtn", chunks=rng.choice([1, 2]),
                    chunk_size=rng.choice([16, 32]), directions=log_int(33, 400))
        most = 12000
    else:
        mode = "fp64" if kind == "far" else rng.choice(["fp32", "tc", "tc", "fp64"])
        size = rng.choice([16, 16, 32, 64] if mode == "tc" else [4, 8, 16, 16, 32])
        chunks = min(chunks, 64 // size)
        case = dict(kind=kind, mode=mode, op="bie" if kind != "apply" else rng.choice(["bie", "bie", "dtn", "all"]),
                    chunks=chunks, chunk_size=size)
        if kind == "apply":
            case["host"] = rng.random() < 0.15
        if kind == "near":
            case["points"] = log_int(500, 60000)
        if kind == "far":
            case["directions"] = log_int(16, 1000)
        # wavenumber groups of 16 columns x triangles^2 weighted by the arithmetic's cost, within the torus case's
        most = math.sqrt(153600.0 ** 2 * 3.5 / ({"fp32": 6, "tc": 1, "fp64": 14}[mode] * chunks * -(-size // 16)))
        most = min(most, 100000)
        if kind == "near":
            most = min(most, 40000)
    if rng.random() < 0.25:
        level = rng.randint(2, 6)
        while 20 * 4 ** level > most:
            level -= 1
        case.update(mesh="sphere", a=level, b=0)
    else:
        # 2 a b triangles, the grid about three times as long as wide
        tri = log_int(300, most)
        a = max(5, int(round(math.sqrt(tri / 6.0) * rng.uniform(0.9, 1.1))))
        case.update(mesh="torus", a=a, b=max(7, tri // (2 * a)))
    return case


# ---- inputs ------------------------------------------------------------------------


def _mesh(case, seed):
    if case["mesh"] == "sphere":
        return sh_perturbed_sphere(case["a"], 5, 0.15, seed)
    coords, tris = torus(1.0, 0.4, case["a"], case["b"])
    return coords * (1.0 + 0.05 * np.random.default_rng(seed).standard_normal(3)), tris


def _coeff(case, kappa):
    """(mass, single layer, double layer, adjoint double layer) per wavenumber."""
    if case["op"] == "bie":
        return np.array([[0.5, -1j * k, 1.0, 0.0] for k in kappa])
    if case["op"] == "dtn":
        return np.array([[0.5, -1j * k, 0.0, 1.0] for k in kappa])
    return np.array([[0.5 + 0.1j, 0.3 - 1j * k, 1.0 + 0.2j, 0.7 - 0.4j] for k in kappa])


def _unit(rng, n):
    d = rng.standard_normal((n, 3))
    return d / np.linalg.norm(d, axis=1, keepdims=True)


def _density(case, seed, coords, kappa):
    """Densities as solves meet them: per column a wave of its wavenumber on the
    surface with a random amplitude, and a rough part."""
    rng = np.random.default_rng(seed + 1)
    size = case["chunk_size"]
    x = torch.from_numpy(coords).cuda()
    gen = torch.Generator(device="cuda").manual_seed(seed)
    out = torch.empty(coords.shape[0], size * len(kappa), dtype=torch.complex128, device="cuda")
    for c, k in enumerate(kappa):
        d = torch.from_numpy(_unit(rng, size)).cuda()
        amp = torch.from_numpy(rng.standard_normal(size) + 1j * rng.standard_normal(size)).cuda()
        out[:, c * size:(c + 1) * size] = torch.exp(1j * k * (x @ d.T)) * amp
    rough = torch.randn(out.shape[0], out.shape[1], 2, dtype=torch.float64, device="cuda", generator=gen)
    return out + 0.1 * torch.view_as_complex(rough)


def _inputs(case, seed):
    """What both the library and the 64-bit values are given."""
    coords, tris = _mesh(case, seed)
    kappa = np.array(WAVENUMBERS[case["chunks"]])
    rng = np.random.default_rng(seed + 2)
    d = dict(coords=coords, tris=tris, kappa=kappa, coeff=_coeff(case, kappa),
             wc=case["chunks"] * case["chunk_size"], meas=fibonacci_sphere(case.get("directions", 64)))
    if case["kind"] in ("apply", "near", "far"):
        d["B"] = _density(case, seed, coords, kappa)
        if case["mode"] != "fp64":
            d["B"] = d["B"].to(torch.complex64)
    if case["kind"] == "near":
        d["points"] = points_off_torus(case["points"], seed=seed) if case["mesh"] == "torus" else \
            _unit(rng, case["points"]) * rng.uniform(1.4, 3.0, (case["points"], 1))
    if case["kind"] in ("request", "adjoint"):
        d["waves"] = _unit(rng, case["chunk_size"])
    if case["kind"] == "adjoint":
        # the residual of the far field, and the normal derivative of the total wave
        # (here in the physical-optics approximation, so that no solve is needed for it)
        shape = (case["directions"], d["wc"])
        d["g"] = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
        nu = coords / np.linalg.norm(coords, axis=1, keepdims=True)
        dn, dx = nu @ d["waves"].T, coords @ d["waves"].T
        d["du_dn"] = np.concatenate([2j * k * dn * np.exp(1j * k * dx) for k in kappa], axis=1)
    return d


def prepare(case, seed):
    d = _inputs(case, seed)
    wc, size = d["wc"], case["chunk_size"]
    if case["kind"] == "request":
        # a slot's context lives across requests and has held another mesh before
        ctx = Helmholtz_CUDA(*sh_perturbed_sphere(2, 5, 0.15, 0), d["meas"])
    else:
        ctx = Helmholtz_CUDA(d["coords"], d["tris"], d["meas"])
    ctx.SetApplyMode(MODES[case["mode"]])
    s = dict(case=case, ctx=ctx, **d)
    if case["kind"] == "apply" and case["host"]:
        s["B"] = d["B"].cpu().numpy()
        s["C"] = np.zeros_like(s["B"])
    elif case["kind"] in ("apply", "near", "far"):
        rows = {"apply": len(d["coords"]), "near": case.get("points"), "far": case.get("directions")}[case["kind"]]
        s["C"] = torch.zeros(rows, wc, dtype=d["B"].dtype, device="cuda")
        ctx.LoadBoundaryOperators_PL(d["kappa"], d["coeff"], wc, size)
        if case["kind"] == "near":
            s["points"] = torch.from_numpy(d["points"]).cuda()
    elif case["kind"] == "request":
        ctx.SetRefinement(REFINEMENTS, INNER_TOL)
        s["F"] = np.zeros((case["directions"], wc), np.complex128)
    else:
        ctx.SetRefinement(REFINEMENTS, INNER_TOL)
        s["Y"] = np.zeros((len(d["coords"]), 3))
    return s


def run(s):
    case, ctx = s["case"], s["ctx"]
    if case["kind"] == "apply":
        if case["host"]:
            return ctx.ApplyBoundaryOperators_PL(1.0, s["B"], 0.0, s["C"], s["kappa"], s["coeff"], s["wc"],
                                                 case["chunk_size"])
        return ctx.ApplyBoundaryOperators_PL(1.0, s["B"], 0.0, s["C"])
    if case["kind"] == "near":
        return ctx.ApplyNearFieldOperators_PL(1.0, s["B"], 0.0, s["C"], s["points"])
    if case["kind"] == "far":
        return ctx.ApplyFarFieldOperators_PL(1.0, s["B"], 0.0, s["C"])
    if case["kind"] == "request":
        ctx.SetMesh(s["coords"], s["tris"])
        return ctx.FarField(s["kappa"], s["waves"], s["F"], WaveType.Plane, CG_TOL, GMRES_TOL)
    return ctx.AdjointDerivative_FF(s["kappa"], s["waves"], s["g"], s["Y"], s["du_dn"], WaveType.Plane, CG_TOL,
                                    GMRES_TOL)[0]


# ---- what a pass cannot do without -----------------------------------------------------


def _mesh_sizes(case):
    if case["mesh"] == "sphere":
        return 10 * 4 ** case["a"] + 2, 20 * 4 ** case["a"]
    return case["a"] * case["b"], 2 * case["a"] * case["b"]


def work(case):
    nv, nt = _mesh_sizes(case)
    wc = case["chunks"] * case["chunk_size"]
    elem = 16 if case["mode"] == "fp64" else 8
    mesh = 24 * nv + 12 * nt
    # per pair: 8 flops per column (a complex multiply-add), about 20 for the kernel entry of a wavenumber
    entry = 8 * wc + 20 * case["chunks"]
    if case["kind"] == "apply":
        return {"bytes": 2 * nv * wc * elem + mesh, "flops": nt * nt * entry}
    if case["kind"] == "near":
        return {"bytes": (nv + case["points"]) * wc * elem + 24 * case["points"] + mesh,
                "flops": nt * case["points"] * entry}
    if case["kind"] == "far":
        return {"bytes": (nv + case["directions"]) * wc * elem + 24 * case["directions"] + mesh,
                "flops": nt * case["directions"] * entry}
    # a solve to 1e-10 takes about 25 applies at these wavenumbers
    block = 16 * nv * wc
    return {"bytes": 25 * 2 * block + 16 * case["directions"] * wc + mesh, "flops": 25 * nt * nt * entry}


# ---- the values in 64 bits ---------------------------------------------------------------


class _Surface:
    """P1 boundary-element operators on the triangle midpoints, in torch float64."""

    def __init__(self, coords, tris):
        p = torch.from_numpy(np.asarray(coords, dtype=np.float64)).cuda()
        self.t = torch.from_numpy(np.asarray(tris, dtype=np.int64)).cuda()
        self.nv, self.nt = p.shape[0], self.t.shape[0]
        x = p[self.t]
        self.mid = x.mean(dim=1)
        cross = 0.5 * torch.linalg.cross(x[:, 1] - x[:, 0], x[:, 2] - x[:, 0])
        self.area = cross.norm(dim=1)
        self.nrm = cross / self.area[:, None]
        # the integral of 1 / |x - midpoint| over the triangle, by its three edges, over the area
        total = torch.zeros_like(self.area)
        for e in range(3):
            a, b = x[:, e] - self.mid, x[:, (e + 1) % 3] - self.mid
            edge = (b - a) / (b - a).norm(dim=1, keepdim=True)
            sa, sb = (a * edge).sum(1), (b * edge).sum(1)
            h = (a - sa[:, None] * edge).norm(dim=1)
            total += h * (torch.asinh(sb / h) - torch.asinh(sa / h))
        self.diag = total / self.area

    def to_triangles(self, V):
        return (self.area / 3).to(V.dtype)[:, None] * V[self.t].sum(dim=1)

    def to_vertices(self, T):
        W = (self.area / 3).to(T.dtype)[:, None] * T
        out = torch.zeros(self.nv, T.shape[1], dtype=T.dtype, device=T.device)
        for q in range(3):
            out.index_add_(0, self.t[:, q], W)
        return out

    def mass(self, V):
        W = self.area.to(V.dtype)[:, None, None] / 12
        X = V[self.t]
        Y = W * (X + X.sum(dim=1, keepdim=True))
        out = torch.zeros_like(V)
        for q in range(3):
            out.index_add_(0, self.t[:, q], Y[:, q])
        return out

    def kernels(self, x, kappa, coeff, nu=None, first=None):
        """Real and imaginary parts of the kernel of each wavenumber, points x against all triangles;
        `first`: x are the midpoints of triangles first, first + 1, ..., the pair itself on the diagonal."""
        z = [self.mid[None, :, q] - x[:, q, None] for q in range(3)]
        r2 = z[0] * z[0] + z[1] * z[1] + z[2] * z[2]
        if first is not None:
            rows = torch.arange(x.shape[0], device=x.device)
            r2[rows, rows + first] = 1.0
        ri = r2.rsqrt_()
        dmu = z[0] * self.nrm[:, 0] + z[1] * self.nrm[:, 1] + z[2] * self.nrm[:, 2]
        dnu = None if nu is None else z[0] * nu[:, 0, None] + z[1] * nu[:, 1, None] + z[2] * nu[:, 2, None]
        del z
        ri3 = ri ** 3
        dmu *= ri3
        if dnu is not None:
            dnu *= ri3
        r = 1.0 / ri
        for k, c in zip(kappa, coeff):
            c1, c2, c3 = (complex(v) / (4 * math.pi) for v in c[1:])
            kr = k * r
            u = (dmu * c2.real, dmu * c2.imag)
            if dnu is not None and c3 != 0:
                u = (u[0] - dnu * c3.real, u[1] - dnu * c3.imag)
            hx = c1.real * ri - u[0] - kr * u[1]   # c1 / r + u (i k r - 1)
            hy = c1.imag * ri - u[1] + kr * u[0]
            cs, sn = torch.cos(kr), torch.sin_(kr)
            re, im = hx * cs - hy * sn, hx * sn + hy * cs
            if first is not None:
                d = c1 * (self.diag[first:first + x.shape[0]] + 1j * k)
                re[rows, rows + first], im[rows, rows + first] = d.real, d.imag
            yield re, im

    def _rows(self):
        return max(16, int(1.5e8) // self.nt)

    def potential(self, x, kappa, coeff, T, nu=None, self_pairs=False):
        """The kernels times a triangle block, its columns in chunks of one wavenumber."""
        size = T.shape[1] // len(kappa)
        out = torch.empty(x.shape[0], T.shape[1], dtype=torch.complex128, device="cuda")
        parts = [torch.cat([T[:, c * size:(c + 1) * size].real, T[:, c * size:(c + 1) * size].imag], 1).contiguous()
                 for c in range(len(kappa))]
        for i in range(0, x.shape[0], self._rows()):
            at = slice(i, min(i + self._rows(), x.shape[0]))
            pairs = self.kernels(x[at], kappa, coeff, None if nu is None else nu[at], i if self_pairs else None)
            for c, (re, im) in enumerate(pairs):
                p, q = re @ parts[c], im @ parts[c]
                out[at, c * size:(c + 1) * size] = torch.complex(p[:, :size] - q[:, size:], p[:, size:] + q[:, :size])
        return out

    def solve(self, kappa, coeff, rhs):
        """The boundary integral equation, by a dense factorisation per wavenumber."""
        size = rhs.shape[1] // len(kappa)
        third = (self.area / 3).to(torch.complex128)
        out = torch.empty_like(rhs)
        for c, k in enumerate(kappa):
            A = torch.zeros(self.nv, self.nv, dtype=torch.complex128, device="cuda")
            for i in range(0, self.nt, self._rows()):
                at = slice(i, min(i + self._rows(), self.nt))
                re, im = next(self.kernels(self.mid[at], [k], [coeff[c]], self.nrm[at], i))
                K = torch.complex(re, im) * third[at, None] * third[None, :]
                W = torch.zeros(K.shape[0], self.nv, dtype=torch.complex128, device="cuda")
                for q in range(3):
                    W.index_add_(1, self.t[:, q], K)
                for q in range(3):
                    A.index_add_(0, self.t[at, q], W)
            w = complex(coeff[c][0]) * self.area.to(torch.complex128) / 12
            for p in range(3):
                for q in range(3):
                    A.index_put_((self.t[:, p], self.t[:, q]), w * (2 if p == q else 1), accumulate=True)
            at = slice(c * size, (c + 1) * size)
            out[:, at] = torch.linalg.solve(A, rhs[:, at])
            del A
        return out

    def far(self, d, kappa, coeff, T):
        size = T.shape[1] // len(kappa)
        out = torch.empty(d.shape[0], T.shape[1], dtype=torch.complex128, device="cuda")
        for c, k in enumerate(kappa):
            c1, c2 = (complex(v) / (4 * math.pi) for v in coeff[c][1:3])
            at = slice(c * size, (c + 1) * size)
            K = (c1 - 1j * k * c2 * (d @ self.nrm.T)) * torch.exp(-1j * k * (d @ self.mid.T))
            out[:, at] = K @ T[:, at]
        return out

    def mass_inverse(self, V):
        M = torch.zeros(self.nv, self.nv, dtype=torch.float64, device="cuda")
        for p in range(3):
            for q in range(3):
                M.index_put_((self.t[:, p], self.t[:, q]), self.area / (6 if p == q else 12), accumulate=True)
        return torch.linalg.solve(M, V)


def exact(case, seed):
    d = _inputs(case, seed)
    S = _Surface(d["coords"], d["tris"])
    kappa, coeff = d["kappa"], d["coeff"]
    if case["kind"] == "apply":
        V = d["B"].to(torch.complex128)
        size = case["chunk_size"]
        C = S.to_vertices(S.potential(S.mid, kappa, coeff, S.to_triangles(V), S.nrm, True))
        c0 = torch.from_numpy(np.repeat(coeff[:, 0], size)).cuda()
        C += c0 * S.mass(V)
        return C.cpu().numpy() if case["host"] else C
    if case["kind"] == "near":
        return S.potential(torch.from_numpy(d["points"]).cuda(), kappa, coeff,
                           S.to_triangles(d["B"].to(torch.complex128)))
    meas = torch.from_numpy(d["meas"]).cuda()
    if case["kind"] == "far":
        return S.far(meas, kappa, coeff, S.to_triangles(d["B"]))
    if S.nv > 12000:
        return None   # the dense factorisation would take too long
    if case["kind"] == "request":
        w = torch.from_numpy(d["waves"]).cuda()
        wave = torch.cat([-torch.exp(1j * k * (S.mid @ w.T)) for k in kappa], 1)
        phi = S.solve(kappa, coeff, S.to_vertices(wave))
        return S.far(meas, kappa, coeff, S.to_triangles(phi)).cpu().numpy()
    # adjoint: Herglotz wave of conj(g) and its normal derivative, the Dirichlet-to-Neumann solve,
    # the product with du/dn along the normals, the mass inverse
    size = case["chunk_size"]
    g = torch.from_numpy(d["g"]).cuda().conj().resolve_conj()
    wave = torch.empty(S.nt, d["wc"], dtype=torch.complex128, device="cuda")
    for c, k in enumerate(kappa):
        at = slice(c * size, (c + 1) * size)
        K = (-1j * k - 1j * k * (S.nrm @ meas.T)) * torch.exp(-1j * k * (S.mid @ meas.T)) / len(meas)
        wave[:, at] = K @ g[:, at]
    dv = S.solve(kappa, coeff, S.to_vertices(wave))
    prod = (torch.from_numpy(d["du_dn"]).cuda() * dv).sum(dim=1, keepdim=True)
    T = S.to_triangles(prod).real / S.area[:, None] * S.nrm * (-1.0 / d["wc"])
    return S.mass_inverse(S.to_vertices(T)).cpu().numpy()
