"""Performance cases: what programs that use this engine have it do.

Each case is one call (or one short chain of calls) through the package's
public entry points: the driver (`CoreManager.run`) on its boundary-value
problems, the operator calls of `Engine`, the sweep's batched assembly, the
dense solvers and the shape gradient.  Sizes are those of the repository's
configurations and tests (icospheres of 80 to 5120 panels, GaussQR 3 to 5,
the latitude-longitude sphere at odd sizes, the 2D disk).  Meshes are spheres
with a smooth radial perturbation of 2 % drawn from the seed, so that another
seed gives another mesh, and the boundary data are the repository's plane wave
and point source.

`exact` evaluates the same quadrature, operators and systems in plain torch
in 64 bits.
"""
from __future__ import annotations

import functools
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for _p in (os.path.join(ROOT, "taichi-bem_b200"), ROOT):
    if _p not in sys.path:
        sys.path.insert(0, _p)

DEV = "cuda"
F64, C128 = torch.float64, torch.complex128


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest solve of the tests: 80 panels, where launches and host work count
        dict(name="dirichlet-80", kind="run", mesh="ico1", kernel="Helmholtz", boundary="Dirichlet",
             scope="Interior", k=2.0, Q=3, precision="fp64"),
        # Laplace interior Dirichlet in the driver's default precision (1280 panels, GaussQR 5)
        dict(name="laplace-1280", kind="run", mesh="ico3", kernel="Laplace", boundary="Dirichlet",
             scope="Interior", k=0.0, Q=5, precision="fp64"),
        # Helmholtz interior Dirichlet at k = 3, 5120 panels, the mixed-precision path
        dict(name="helmholtz-5120-mixed", kind="run", mesh="ico4", kernel="Helmholtz", boundary="Dirichlet",
             scope="Interior", k=3.0, Q=5, precision="mixed"),
        # exterior Neumann problem on a ragged mesh: hypersingular block, adjoint double layer in the right-hand side
        dict(name="neumann-990", kind="run", mesh="uv16x33", kernel="Helmholtz", boundary="Neumann",
             scope="Exterior", k=2.5, Q=4, precision="fp64"),
        # transmission least squares (k_in = 1.5 k_out) in mixed precision: 7682 unknowns
        dict(name="transmission-5120-mixed", kind="run", mesh="ico4", kernel="Helmholtz_Transmission",
             boundary="Full", scope="Exterior", k=5.0, Q=4, precision="mixed"),
        # the same on the plain path, ragged (2070 panels, 3107 unknowns)
        dict(name="transmission-2070", kind="run", mesh="uv24x45", kernel="Helmholtz_Transmission",
             boundary="Full", scope="Exterior", k=5.0, Q=4, precision="fp64"),
        # one dense operator block, the unit of every program that brings its own solver
        dict(name="single-layer-5120", kind="assemble", mesh="ico4", op="V", k=3.0, Q=5, precision="fp64"),
        # matrix-free product of the Laplace double layer (right-hand sides)
        dict(name="double-layer-apply-2970", kind="apply", mesh="uv34x45", op="K", k=0.0, Q=5, precision="fp64"),
        # the wavenumber sweep's batched assembly: P1/P1 operators of two media at four k
        dict(name="sweep-operators-1280", kind="sweep", mesh="ico3", k=16.0, nk=4, Q=3, precision="mixed"),
        # least squares of a sweep step: normal matrix, Cholesky, FP64 flexible GMRES, 2 right-hand sides
        dict(name="lstsq-2999-mixed", kind="lstsq", n=2999, nrhs=2, precision="mixed"),
        # dense FP64 factorisation with partial pivoting and solves (the default solver)
        dict(name="lu-2999-complex", kind="lu", n=2999, nrhs=3, dtype="complex128"),
        # shape gradient: forward solve and adjoint of the Laplace problem through autograd
        dict(name="shape-5120-mixed", kind="shape", mesh="ico4", Q=4, precision="mixed"),
    ]


def draw(rng):
    def log_between(a, b):
        return math.exp(rng.uniform(math.log(a), math.log(b)))

    def ragged(a, b):
        """A latitude-longitude sphere of about log-uniformly many panels."""
        nt = log_between(a, b)
        rows = max(4, int(round(math.sqrt(nt / 2.0 / rng.uniform(1.1, 1.7)))))
        cols = max(5, int(round(nt / (2.0 * (rows - 1)))))
        return f"uv{rows}x{cols}"

    kind = rng.choice(["run", "run", "run", "transmission", "assemble", "apply", "sweep", "lstsq", "lu", "shape"])
    precision = rng.choice(["fp64", "mixed"])
    k = round(rng.uniform(0.8, 2.6), 3)
    Q = rng.choice([3, 4, 5])
    if kind == "run":
        kernel = rng.choice(["Laplace", "Helmholtz", "Helmholtz"])
        boundary = "Dirichlet" if kernel == "Laplace" else rng.choice(["Dirichlet", "Dirichlet", "Neumann"])
        scope = "Interior" if boundary == "Dirichlet" else "Exterior"
        return dict(kind="run", mesh=ragged(60, 4500), kernel=kernel, boundary=boundary, scope=scope,
                    k=0.0 if kernel == "Laplace" else k, Q=Q, precision=precision)
    if kind == "transmission":
        return dict(kind="run", mesh=ragged(100, 2100), kernel="Helmholtz_Transmission", boundary="Full",
                    scope="Exterior", k=round(rng.uniform(1.0, 6.0), 3), Q=Q, precision=precision)
    if kind == "assemble":
        return dict(kind="assemble", mesh=ragged(200, 5000), op=rng.choice(["V", "K", "W"]),
                    k=rng.choice([0.0, round(rng.uniform(0.5, 8.0), 3)]), Q=Q, precision=precision)
    if kind == "apply":
        return dict(kind="apply", mesh=ragged(200, 5000), op=rng.choice(["V", "K", "KP", "W"]),
                    k=rng.choice([0.0, round(rng.uniform(0.5, 8.0), 3)]), Q=Q, precision=precision)
    if kind == "sweep":
        return dict(kind="sweep", mesh=ragged(100, 1400), k=round(rng.uniform(3.0, 18.0), 3), nk=rng.choice([1, 2, 3, 4]),
                    Q=3, precision=precision)
    if kind == "lstsq":
        return dict(kind="lstsq", n=int(log_between(200, 3000)), nrhs=rng.choice([1, 2, 4]), precision=precision)
    if kind == "lu":
        return dict(kind="lu", n=int(log_between(100, 3000)), nrhs=rng.choice([1, 2, 3]),
                    dtype=rng.choice(["complex128", "float64"]))
    # the shape problem needs a mesh without slivers
    return dict(kind="shape", mesh=rng.choice(["ico2", "ico3", "ico3"]), amplitude=round(rng.uniform(0.005, 0.04), 4),
                Q=Q, precision=precision)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _base_mesh(name):
    from bem_b200.meshes import analytical_sphere, icosphere
    if name.startswith("ico"):
        return icosphere(int(name[3:]))
    rows, cols = (int(x) for x in name[2:].split("x"))
    return analytical_sphere(1.0, rows, cols)


def mesh_of(case, seed):
    """The base sphere with a seeded smooth radial perturbation (2 % unless
    the case says otherwise)."""
    v, f = _base_mesh(case["mesh"])
    rng = np.random.default_rng(seed)
    w = rng.standard_normal((6, 3)) * 2.0
    delta = np.sin(v @ w.T + rng.uniform(0.0, 2.0 * math.pi, 6)) @ rng.standard_normal(6)
    delta *= case.get("amplitude", 0.02) / np.abs(delta).max()
    return v * (1.0 + delta)[:, None], f


def _direction(seed):
    g = np.random.default_rng(seed + 1000003).standard_normal(3)
    return g / np.linalg.norm(g)


def _source(seed):
    return tuple(2.0 + np.random.default_rng(seed + 1000003).uniform(-0.3, 0.3, 3))


def _params(case, v, f):
    deg = case.get("degree", 0)
    return dict(dim=3, object="generated", vertices=v, panels=f, GaussQR=case["Q"], kernel=case["kernel"], k=case["k"],
                boundary=case["boundary"], scope=case["scope"], n_i=case.get("n_i", 2.25), n_o=1.0, Q_Neumann=deg,
                Q_Dirichlet=1, show="Default", precision=case["precision"])


def _manager(case, seed):
    from bem_b200.managers import CoreManager
    from bem_b200.workloads import laplace_point_source, plane_wave
    v, f = mesh_of(case, seed)
    fD, fN = laplace_point_source(_source(seed)) if case["kernel"] == "Laplace" else plane_wave(case["k"],
                                                                                            _direction(seed))
    core = CoreManager(_params(case, v, f))
    core.initialization(fD, fN)
    return core


def _sweep_case(case):
    return dict(case, kernel="Helmholtz_Transmission", boundary="Full", scope="Exterior", n_i=3.0, degree=1)


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _randn(shape, dtype, g):
    x = torch.randn(shape, dtype=F64, device=DEV, generator=g)
    return torch.complex(x, torch.randn(shape, dtype=F64, device=DEV, generator=g)) if dtype == C128 else x


def _dense_inputs(case, seed):
    """Dense systems with the decay and the diagonal of a discretised
    operator: a smooth kernel between random points of the sphere, a random
    part of a few per cent and a shifted diagonal."""
    n = case["n"]
    dtype = getattr(torch, case.get("dtype", "complex128"))
    g = _gen(seed)
    x = torch.randn(n, 3, dtype=F64, device=DEV, generator=g)
    x = x / x.norm(dim=1, keepdim=True)
    r = torch.cdist(x, x) + 0.05

    def matrix(k):
        A = torch.exp(1j * k * r) / r if dtype == C128 else torch.cos(k * r) / r
        A = A / n + 0.02 * _randn((n, n), dtype, g) / math.sqrt(n)
        return (A + 0.2 * torch.eye(n, dtype=dtype, device=DEV)).contiguous()

    A = matrix(3.0)
    P = matrix(4.5) if case["kind"] == "lstsq" else None
    m = 2 * n if case["kind"] == "lstsq" else n
    return A, P, _randn((m, case["nrhs"]), dtype, g)


_OPS = {"V": 0, "K": 1, "KP": 2, "W": 3}
_DEGREE = {"V": (1, 1), "K": (1, 3), "KP": (3, 1), "W": (3, 3)}  # bases per panel of the test and trial spaces


def _operator_state(case, seed):
    from bem_b200 import _lib as L
    from bem_b200.engine import DeviceSpace, Engine
    v, f = mesh_of(case, seed)
    eng = Engine(DEV)
    eng.set_mesh(v, f, case["Q"])
    ids = np.arange(len(f), dtype=np.int32)
    space = {1: lambda: DeviceSpace.from_numpy(ids, 1, ids, eng.device),
             3: lambda: DeviceSpace.from_numpy(ids, 3, f.reshape(-1).copy(), eng.device)}
    nbx, nby = _DEGREE[case["op"]]
    test, trial = space[nbx](), space[nby]()
    if nbx == nby:
        trial = test
    rows, cols = (len(f) if nb == 1 else len(v) for nb in (nbx, nby))
    helm = case["k"] > 0
    desc = Engine.op_desc(_OPS[case["op"]], helm, case["k"], case["k"] ** 2, quirk=True,
                          precision=L.PREC_MIXED if case["precision"] == "mixed" else L.PREC_FP64)
    dtype = C128 if helm else F64
    st = dict(kind=case["kind"], engine=eng, desc=desc, test=test, trial=trial)
    if case["kind"] == "assemble":
        st["out"] = torch.zeros(rows, cols, dtype=dtype, device=DEV)
    else:
        st["x"] = _randn(cols, dtype, _gen(seed))
        st["y"] = torch.zeros(rows, dtype=dtype, device=DEV)
    return st


def prepare(case, seed):
    kind = case["kind"]
    if kind == "run":
        return dict(kind="run", core=_manager(case, seed))
    if kind in ("assemble", "apply"):
        return _operator_state(case, seed)
    if kind == "sweep":
        return dict(kind="sweep", core=_manager(_sweep_case(case), seed),
                    ks=[case["k"] + i / 30.0 for i in range(case["nk"])])
    if kind == "lstsq":
        from bem_b200.engine import Engine
        A, P, B = _dense_inputs(case, seed)
        return dict(kind="lstsq", engine=Engine(DEV), A=A, P=P, B=B, mixed=case["precision"] == "mixed")
    if kind == "lu":
        from bem_b200.engine import Engine
        A, _, B = _dense_inputs(case, seed)
        return dict(kind="lu", engine=Engine(DEV), A=A, B=B)
    if kind == "shape":
        from bem_b200.shape import DirichletShape, point_source
        v, f = mesh_of(case, seed)
        u, gu = point_source(_source(seed))
        prob = DirichletShape(f, u, gu, gauss_qr=case["Q"], precision=case["precision"])
        X = torch.as_tensor(v, device=DEV).requires_grad_(True)
        target = torch.randn(len(f), dtype=F64, device=DEV, generator=_gen(seed))
        return dict(kind="shape", problem=prob, X=X, target=target)
    raise ValueError(kind)


def run(state):
    kind = state["kind"]
    if kind == "run":
        core = state["core"]
        core.run()
        b = core._BEM_manager
        return {"raw_solved": b.raw_solved, "solved": b.solved}
    if kind == "assemble":
        state["out"].zero_()
        state["engine"].assemble(state["desc"], state["test"], state["trial"], state["out"])
        return state["out"]
    if kind == "apply":
        state["y"].zero_()
        state["engine"].apply(state["desc"], state["test"], state["trial"], state["x"], state["y"])
        return state["y"]
    if kind == "sweep":
        from bem_b200.managers.sweep import transmission_operators
        return transmission_operators(state["core"]._BEM_manager, state["ks"])
    if kind == "lstsq":
        eng, A, P, B = state["engine"], state["A"], state["P"], state["B"]
        n = A.shape[0]
        N = torch.empty_like(A)
        d = torch.empty(n, dtype=F64, device=DEV)
        eng.gram(A, P, N, d, tensor_cores=state["mixed"])
        piv, dinv, _ = eng.chol_factor(N, tensor_cores=state["mixed"])
        X = torch.zeros(n, B.shape[1], dtype=A.dtype, device=DEV)
        for c in range(B.shape[1]):
            x = torch.zeros(n, dtype=A.dtype, device=DEV)
            eng.lstsq_refine(A, P, d, N, piv, dinv, B[:, c].contiguous(), x)
            X[:, c] = x
        return X
    if kind == "lu":
        eng, B = state["engine"], state["B"]
        LU = state["A"].clone()
        piv, _ = eng.lu_factor(LU)
        return eng.lu_solve(LU, piv, B.clone())
    if kind == "shape":
        from bem_b200.shape import DirichletShapeSolve
        X = state["X"]
        X.grad = None
        t = DirichletShapeSolve.apply(X, state["problem"])
        ((t - state["target"]) ** 2).sum().backward()
        return {"t": t.detach(), "grad": X.grad}
    raise ValueError(kind)


# ---------------------------------------------------------------------------
# the work of one pass
# ---------------------------------------------------------------------------
def work(case):
    """Floating-point operations of the quadrature (every pair of points of
    every pair of panels once: distance, reciprocal root, and for Helmholtz
    the exponential, some 20 and 40 operations) and of the dense solve, and
    the bytes of the blocks written and read once."""
    kind = case["kind"]
    if kind in ("lstsq", "lu"):
        n, c = case["n"], 8.0 if case.get("dtype", "complex128") == "complex128" else 2.0
        b = 2.0 * c
        if kind == "lu":
            return {"bytes": 2.0 * b * n * n, "flops": c * n ** 3 / 3.0}
        return {"bytes": 3.0 * 16 * n * n, "flops": 8.0 * n ** 3 + 8.0 * n ** 3 / 6.0}
    v, f = _base_mesh(case["mesh"])
    nt, nv, Q4 = len(f), len(v), float(case["Q"]) ** 4
    helm = case.get("k", 0.0) > 0
    per, b = (40.0, 16.0) if helm else (20.0, 8.0)
    if kind == "assemble":
        rows, cols = (nt if nb == 1 else nv for nb in _DEGREE[case["op"]])
        sym = 0.5 if case["op"] in ("V", "W") else 1.0
        return {"bytes": b * rows * cols, "flops": sym * per * nt * nt * Q4}
    if kind == "apply":
        rows, cols = (nt if nb == 1 else nv for nb in _DEGREE[case["op"]])
        sym = 0.5 if case["op"] in ("V", "W") else 1.0
        return {"bytes": b * (rows + cols) + 100.0 * nt, "flops": sym * per * nt * nt * Q4}
    if kind == "sweep":
        return {"bytes": case["nk"] * 2.0 * 16 * (2.0 * nv) ** 2, "flops": case["nk"] * 2 * 0.5 * 80 * nt * nt * Q4}
    if kind == "shape":
        return {"bytes": 2.0 * 8 * nt * nt, "flops": 4 * 0.5 * 20.0 * nt * nt * Q4 + 2.0 * nt ** 3 / 3.0}
    if case["kernel"] == "Helmholtz_Transmission":
        n = nt + nv
        return {"bytes": 3.0 * 16 * n * n,
                "flops": 2 * 0.5 * 80 * nt * nt * Q4 + 8.0 * n ** 3 + 8.0 * n ** 3 / 6.0}
    n = nt if case["boundary"] == "Dirichlet" else nv
    return {"bytes": 2 * b * n * n, "flops": 0.5 * 1.5 * per * nt * nt * Q4 + (8.0 if helm else 2.0) * n ** 3 / 3.0}


# ---------------------------------------------------------------------------
# the same quantities in plain torch, 64 bits
# ---------------------------------------------------------------------------
class _Quadrature:
    """Galerkin blocks on a triangle mesh: the collapsed GaussQR^4 rule on
    separate panels, its coincident / edge / vertex maps on touching ones."""

    def __init__(self, v, f, Q):
        self.X = v if isinstance(v, torch.Tensor) else torch.as_tensor(np.ascontiguousarray(v), device=DEV)
        self.f = torch.as_tensor(np.asarray(f, np.int64), device=DEV)
        self.nt, self.nv = len(f), len(self.X)
        p, w = np.polynomial.legendre.leggauss(Q)
        self.gp, self.gw = (p + 1.0) / 2.0, w / 2.0
        r1 = np.repeat(self.gp, Q)
        r2 = r1 * np.tile(self.gp, Q)
        self.bary = torch.as_tensor(np.stack([1 - r1, r1 - r2, r2], 1), device=DEV)  # [Q2, 3]
        self.w = torch.as_tensor(np.repeat(self.gw, Q) * np.tile(self.gw, Q) * r1, device=DEV)
        share = torch.zeros(self.nt, self.nt, dtype=torch.int8, device=DEV)
        for a in range(3):
            for b in range(3):
                share += (self.f[:, a, None] == self.f[None, :, b]).to(torch.int8)
        self.share = share
        self.geometry()

    def geometry(self):
        P = self.X[self.f]  # [nt, 3, 3]
        cr = torch.linalg.cross(P[:, 1] - P[:, 0], P[:, 2] - P[:, 1])
        J = torch.linalg.norm(cr, dim=1)
        self.P, self.J, self.n = P, J, cr / J[:, None]  # J = 2 area
        opp = torch.stack([P[:, 2] - P[:, 1], P[:, 0] - P[:, 2], P[:, 1] - P[:, 0]], 1)
        g = torch.linalg.cross(self.n[:, None, :].expand(-1, 3, -1), opp) / J[:, None, None]
        self.curl = torch.linalg.cross(self.n[:, None, :].expand(-1, 3, -1), g)
        self.pts = torch.einsum("qb,tbc->tqc", self.bary, P)

    # kernel value: op over d = x - y, real and imaginary part (None for Laplace)
    @staticmethod
    def value(op, d, nx, ny, k):
        r2 = (d * d).sum(-1)
        r = r2.sqrt()
        if op in ("V", "W"):
            t = 1.0 / r
            if k == 0:
                return t, None
            return t * torch.cos(k * r), t * torch.sin(k * r)
        dn = (d * ny).sum(-1) if op == "K" else -(d * nx).sum(-1)
        t = dn / (r2 * r)
        if k == 0:
            return t, None
        kr = k * r
        c, s = torch.cos(kr), torch.sin(kr)
        return t * (c + kr * s), t * (s - kr * c)

    def basis(self, nb, bary):
        return torch.ones_like(bary[..., :1]) if nb == 1 else bary

    def combine(self, op, k, k2, i, j, mom0, momb):
        """Entries from the plain and the basis-weighted moments of pairs."""
        if op != "W":
            return momb
        cd = torch.einsum("...xc,...yc->...xy", self.curl[i], self.curl[j])
        nd = (self.n[i] * self.n[j]).sum(-1)
        return mom0[..., None, None] * cd - (k2 * nd[..., None, None] * momb if k2 else 0.0)

    def far(self, op, k, nbx, nby, i0, i1):
        """[c, nbx, nt, nby] values of test panels i0..i1 against all panels
        (zero where the panels touch)."""
        i = torch.arange(i0, i1, device=DEV)
        d = self.pts[i][:, :, None, None, :] - self.pts[None, None, :, :, :]  # [c, Q2, nt, Q2, 3]
        sep = (self.share[i0:i1] == 0)
        d = torch.where(sep[:, None, :, None, None], d, torch.ones_like(d))  # d = 0 on a panel with itself
        parts = self.value(op, d, self.n[i][:, None, None, None, :], self.n[None, None, :, None, :], k)
        scale = self.J[i][:, None] * self.J[None, :] * sep / (4 * math.pi)
        wx = self.w[:, None] * self.basis(nbx, self.bary)
        wy = self.w[:, None] * self.basis(nby, self.bary)
        out = []
        for part in parts:
            if part is None:
                continue
            part = torch.where(sep[:, None, :, None], part, torch.zeros_like(part))
            m = torch.einsum("cajb,by->cajy", part, wy)
            momb = torch.einsum("cajy,ax->cjxy", m, wx) * scale[..., None, None]
            mom0 = None
            if op == "W":
                mom0 = torch.einsum("cajb,a,b->cj", part, self.w, self.w) * scale
            out.append((mom0, momb))
        return out

    def near_rule(self, rel):
        """[P] arrays (bary x, bary y, weight, swapped) of one relation."""
        g, w = self.gp, self.gw
        xs, e1, e2, e3 = (a.reshape(-1) for a in np.meshgrid(g, g, g, g, indexing="ij"))
        W = np.prod([a.reshape(-1) for a in np.meshgrid(w, w, w, w, indexing="ij")], axis=0)
        rows = []

        def add(r1x, r2x, r1y, r2y, jac, second=0.0):
            rows.append((r1x, r2x, r1y, r2y, W * jac, np.full_like(W, second)))

        if rel == "coincide":
            jac = xs ** 3 * e1 ** 2 * e2
            w0, w1, w2, w3 = xs, xs * e1, xs * e1 * e2, xs * e1 * e2 * e3
            for z in ((w0, w0 - w1 + w2, w3, w2), (w0, w1 - w2 + w3, w2, w3), (w0 - w3, w1 - w3, -w3, w2 - w3)):
                for second in (0.0, 1.0):
                    add(z[0], z[1], z[0] - z[2], z[1] - z[3], jac, second)
        elif rel == "vertex":
            jac = xs ** 3 * e2
            add(xs, xs * e1, xs * e2, xs * e2 * e3, jac)
            add(xs * e2, xs * e2 * e3, xs, xs * e1, jac)
        else:
            jac1 = xs ** 3 * e1 ** 2
            jac = jac1 * e2
            add(xs, xs * e1 * e3, xs - xs * e1 * e2, xs * e1 * (1 - e2), jac1)
            add(xs, xs * e1, xs - xs * e1 * e2 * e3, xs * e1 * e2 * (1 - e3), jac)
            add(xs * (1 - e1 * e2), xs * e1 * (1 - e2), xs, xs * e1 * e2 * e3, jac)
            add(xs * (1 - e1 * e2 * e3), xs * e1 * e2 * (1 - e3), xs, xs * e1, jac)
            add(xs * (1 - e1 * e2 * e3), xs * e1 * (1 - e2 * e3), xs, xs * e1 * e2, jac)
        r1x, r2x, r1y, r2y, wt, sec = (np.concatenate(c) for c in zip(*rows))
        T = lambda a: torch.as_tensor(a, device=DEV)
        return (T(np.stack([1 - r1x, r1x - r2x, r2x], 1)), T(np.stack([1 - r1y, r1y - r2y, r2y], 1)), T(wt),
                T(1.0 - 2.0 * sec))

    def near(self, op, k, nbx, nby):
        """(i, j, parts) of the touching pairs, in chunks."""
        for rel, count in (("coincide", 3), ("edge", 2), ("vertex", 1)):
            bx, by, wt, sgn = self.near_rule(rel)
            pairs = (self.share == count).nonzero()
            step = max(1, 3_000_000 // len(wt))
            for c0 in range(0, len(pairs), step):
                i, j = pairs[c0:c0 + step].unbind(1)
                d = torch.einsum("pb,mbc->mpc", bx, self.P[i]) - torch.einsum("pb,mbc->mpc", by, self.P[j])
                if op in ("K", "KP"):
                    d = d * sgn[None, :, None]
                parts = self.value(op, d, self.n[i][:, None, :], self.n[j][:, None, :], k)
                scale = self.J[i] * self.J[j] / (4 * math.pi)
                out = []
                for part in parts:
                    if part is None:
                        continue
                    part = part * wt * scale[:, None]
                    momb = torch.einsum("mp,px,py->mxy", part, self.basis(nbx, bx), self.basis(nby, by))
                    out.append((part.sum(1) if op == "W" else None, momb))
                yield i, j, out

    def chunk(self):
        return max(1, 3_000_000 // (len(self.w) ** 2 * self.nt))

    def block(self, op, k=0.0, nbx=1, nby=1, k2=None):
        """The dense block of op; dofs: panels (nb = 1) or vertices (nb = 3)."""
        k2 = k * k if k2 is None else k2
        size = {1: self.nt, 3: self.nv}
        dof = {1: torch.arange(self.nt, device=DEV)[:, None], 3: self.f}
        parts = [torch.zeros(size[nbx], size[nby], dtype=F64, device=DEV) for _ in range(1 if k == 0 else 2)]
        allj = torch.arange(self.nt, device=DEV)
        step = self.chunk()
        for i0 in range(0, self.nt, step):
            i1 = min(self.nt, i0 + step)
            i = torch.arange(i0, i1, device=DEV)
            for out, (mom0, momb) in zip(parts, self.far(op, k, nbx, nby, i0, i1)):
                e = self.combine(op, k, k2, i[:, None], allj[None, :], mom0, momb)  # [c, nt, nbx, nby]
                tmp = torch.zeros((i1 - i0) * nbx, size[nby], dtype=F64, device=DEV)
                tmp.index_add_(1, dof[nby].reshape(-1), e.permute(0, 2, 1, 3).reshape((i1 - i0) * nbx, -1))
                out.index_add_(0, dof[nbx][i].reshape(-1), tmp)
        for i, j, vals in self.near(op, k, nbx, nby):
            for out, (mom0, momb) in zip(parts, vals):
                e = self.combine(op, k, k2, i, j, mom0, momb)
                r = dof[nbx][i][:, :, None].expand(-1, -1, nby)
                c = dof[nby][j][:, None, :].expand(-1, nbx, -1)
                out.index_put_((r.reshape(-1), c.reshape(-1)), e.reshape(-1), accumulate=True)
        return parts[0] if k == 0 else torch.complex(parts[0], parts[1])

    def mass(self, nbx, nby):
        size = {1: self.nt, 3: self.nv}
        dof = {1: torch.arange(self.nt, device=DEV)[:, None], 3: self.f}
        loc = torch.einsum("q,qx,qy->xy", self.w, self.basis(nbx, self.bary), self.basis(nby, self.bary))
        e = self.J[:, None, None] * loc
        out = torch.zeros(size[nbx], size[nby], dtype=F64, device=DEV)
        r = dof[nbx][:, :, None].expand(-1, -1, nby)
        c = dof[nby][:, None, :].expand(-1, nbx, -1)
        return out.index_put_((r.reshape(-1), c.reshape(-1)), e.reshape(-1), accumulate=True)


def _data(case, seed):
    """Boundary data at points x with normals n, wavenumber factor s."""
    if case["kernel"] == "Laplace":
        x0 = torch.tensor(_source(seed), dtype=F64, device=DEV)
        fD = lambda x, s=1.0: 1.0 / torch.linalg.norm(x - x0, dim=1)
        fN = lambda x, n, s=1.0: -((x - x0) * n).sum(1) / torch.linalg.norm(x - x0, dim=1) ** 3
        return fD, fN
    d = torch.as_tensor(_direction(seed), device=DEV)
    k = case["k"]
    fD = lambda x, s=1.0: torch.exp(1j * (k * s) * (x @ d))
    fN = lambda x, n, s=1.0: 1j * (k * s) * (n @ d) * torch.exp(1j * (k * s) * (x @ d))
    return fD, fN


def _exact_run(case, seed):
    v, f = mesh_of(case, seed)
    q = _Quadrature(v, f, case["Q"])
    k = case["k"] if case["kernel"] != "Laplace" else 0.0
    fD, fN = _data(case, seed)
    cent = q.P.mean(1)
    conj = (lambda x: x.conj().resolve_conj()) if k else (lambda x: x)
    cplx = lambda M: M.to(C128) if k else M
    if case["kernel"] == "Helmholtz_Transmission":
        si, so = math.sqrt(case.get("n_i", 2.25)), 1.0
        nv, n = q.nv, q.nv + q.nt

        def half_and(kk, c):
            A = torch.zeros(n, n, dtype=C128, device=DEV)
            V, K, W = q.block("V", kk), q.block("K", kk, 1, 3), q.block("W", kk, 3, 3)
            M = 0.5 * q.mass(1, 3)
            A[nv:, nv:] = -c * V
            A[nv:, :nv] = c * K + M
            A[:nv, nv:] = (-c * K + M).T
            A[:nv, :nv] = -c * W
            return A

        f_b = torch.cat([fD(q.X, si) - fD(q.X, so), fN(cent, q.n, si) - fN(cent, q.n, so)])
        Po = half_and(k * so, -1.0)
        rhs = Po @ conj(f_b)
        P = half_and(k * si, 1.0)
        S = torch.cat([Po + P, P])
        x = torch.linalg.lstsq(S, torch.cat([rhs, torch.zeros_like(rhs)])[:, None]).solution[:, 0]
        return {"raw_solved": x, "solved": None}
    half = 0.5 if case["scope"] == "Interior" else -0.5
    if case["boundary"] == "Dirichlet":
        g = conj(fD(q.X))
        b = half * (cplx(q.mass(1, 3)) @ g) + q.block("K", k, 1, 3) @ g
        x = torch.linalg.solve(q.block("V", k), b)
        va = torch.zeros(q.nv, dtype=F64, device=DEV).index_add_(0, q.f.reshape(-1),
                                                                 (q.J / 6.0).repeat_interleave(3))
        s = torch.zeros(q.nv, dtype=x.dtype, device=DEV)
        s.index_add_(0, q.f.reshape(-1), ((q.J / 6.0)[:, None] / va[q.f] * x[:, None]).reshape(-1))
        return {"raw_solved": x, "solved": s}
    g = conj(fN(cent, q.n))
    b = half * (cplx(q.mass(3, 1)) @ g) - q.block("KP", k, 3, 1) @ g
    return {"raw_solved": torch.linalg.solve(q.block("W", k, 3, 3), b), "solved": None}


def _exact_sweep(case, seed):
    case = _sweep_case(case)
    v, f = mesh_of(case, seed)
    q = _Quadrature(v, f, case["Q"])
    nv, outs = q.nv, []
    M = 0.5 * q.mass(3, 3)

    def operator(kk, c):
        A = torch.zeros(2 * nv, 2 * nv, dtype=C128, device=DEV)
        V, K, W = q.block("V", kk, 3, 3), q.block("K", kk, 3, 3), q.block("W", kk, 3, 3)
        A[nv:, nv:], A[nv:, :nv], A[:nv, nv:], A[:nv, :nv] = -c * V, c * K, -c * K.T, -c * W
        return A

    Id = torch.zeros(2 * nv, 2 * nv, dtype=C128, device=DEV)
    Id[nv:, :nv], Id[:nv, nv:] = M.to(C128), M.T.to(C128)
    for i in range(case["nk"]):
        k = case["k"] + i / 30.0
        P = operator(k * math.sqrt(case["n_i"]), 1.0)
        outs.append(torch.cat([operator(k, -1.0) - P, P + Id]))
    return outs


def _exact_shape(case, seed):
    v, f = mesh_of(case, seed)
    x0 = torch.tensor(_source(seed), dtype=F64, device=DEV)
    target = torch.randn(len(f), dtype=F64, device=DEV, generator=_gen(seed))
    q = _Quadrature(v, f, case["Q"])
    g = 1.0 / torch.linalg.norm(q.X - x0, dim=1)
    V, K, M = q.block("V"), q.block("K", 0.0, 1, 3), q.mass(1, 3)
    t = torch.linalg.solve(V, K @ g + 0.5 * (M @ g))
    lam = torch.linalg.solve(V.T, 2.0 * (t - target))
    # gradient of lam . (K g + M g / 2 - V t) in the vertices, lam and t held
    X = q.X.clone().requires_grad_(True)
    q.X = X

    def fresh():
        q.geometry()
        return (1.0 / torch.linalg.norm(X - x0, dim=1))[q.f]  # [nt, 3]

    loc = torch.einsum("q,qy->y", q.w, q.bary)
    gt = fresh()
    (0.5 * (lam * q.J * (gt @ loc)).sum()).backward()
    step = max(1, q.chunk() // 2)
    for i0 in range(0, q.nt, step):
        i1 = min(q.nt, i0 + step)
        gt = fresh()
        li = lam[i0:i1, None]
        s = -(li * q.far("V", 0.0, 1, 1, i0, i1)[0][1][:, :, 0, 0] * t).sum()
        s = s + (li[:, :, None] * q.far("K", 0.0, 1, 3, i0, i1)[0][1][:, :, 0, :] * gt).sum()
        s.backward()
    for op, nby in (("V", 1), ("K", 3)):
        gt = fresh()
        total = X.new_zeros(())
        for n, (i, j, vals) in enumerate(q.near(op, 0.0, 1, nby)):
            e = vals[0][1][:, 0, :]
            total = total + (lam[i, None] * e * (gt[j] if op == "K" else -t[j, None])).sum()
        total.backward()
    return {"t": t, "grad": X.grad}


def exact(case, seed):
    kind = case["kind"]
    if kind == "run":
        return _exact_run(case, seed)
    if kind in ("assemble", "apply"):
        v, f = mesh_of(case, seed)
        q = _Quadrature(v, f, case["Q"])
        A = q.block(case["op"], case["k"], *_DEGREE[case["op"]])
        if kind == "assemble":
            return A
        return A @ _randn(A.shape[1], A.dtype, _gen(seed))
    if kind == "sweep":
        return _exact_sweep(case, seed)
    if kind == "lstsq":
        A, P, B = _dense_inputs(case, seed)
        return torch.linalg.lstsq(torch.cat([A, P]), B).solution
    if kind == "lu":
        A, _, B = _dense_inputs(case, seed)
        return torch.linalg.solve(A, B)
    if kind == "shape":
        return _exact_shape(case, seed)
    return None
