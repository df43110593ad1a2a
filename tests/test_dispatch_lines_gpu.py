"""Both sides of the lines at which products and solves change kernels,
against numpy or torch in FP64."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    from bem_b200.engine import Engine
    e = Engine()
    yield e
    e.close()


def _gaussian(shape, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*shape, dtype=dtype, device="cuda", generator=g)


_DTYPES = [torch.float64, torch.complex128, torch.float32, torch.complex64]


@pytest.mark.parametrize("dtype", _DTYPES)
@pytest.mark.parametrize("m,n,offset", [(3, 1, 0), (9, 127, 0), (9, 128, 1), (40, 255, 0), (17, 256, 1), (300, 257, 0),
                                        (700, 1024, 0), (65, 1300, 1)])
def test_products_over_chunks(engine, m, n, offset, dtype):
    """Rows of no, one and several chunks with remainders, each row starting at
    its own chunk, a leading dimension beyond n, operands that start `offset`
    elements past an aligned address (complex FP32: 8 bytes).  FP64 sums of n
    products: sqrt(n) roundings of 1.1e-16 of the sum of magnitudes, times 4."""
    hi = torch.complex128 if dtype.is_complex else torch.float64
    A = _gaussian((m * (n + 5) + offset,), dtype, n)[offset:].view(m, n + 5)[:, :n]
    x = _gaussian((n + offset,), hi, 1)[offset:]
    y0 = _gaussian((m,), hi, 2)
    y = y0.clone()
    engine.gemv(A, x, y, alpha=-0.5, beta=2.0)
    Ah = A.to(hi)
    ref = -0.5 * (Ah @ x) + 2.0 * y0
    mag = 0.5 * (Ah.abs() @ x.abs()) + 2.0 * y0.abs()
    assert bool(((y - ref).abs() <= 4 * (n ** 0.5 + 2) * 1.2e-16 * mag).all())


@pytest.mark.parametrize("dtype", [torch.float64, torch.complex128])
def test_product_beyond_the_l2_cache(engine, dtype):
    """Streaming loads: a matrix of more than 126 MB; bound as above."""
    n = 4500 if dtype == torch.float64 else 3300
    A, x = _gaussian((n, n), dtype, 3), _gaussian((n,), dtype, 4)
    y = torch.zeros(n, dtype=dtype, device="cuda")
    engine.gemv(A, x, y)
    assert bool(((y - A @ x).abs() <= 4 * n ** 0.5 * 1.2e-16 * (A.abs() @ x.abs())).all())


@pytest.mark.parametrize("dtype", [torch.float64, torch.complex128])
@pytest.mark.parametrize("conj_a,conj_b", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("m,n,k", [(1290, 1283, 511), (1290, 1283, 512), (1283, 1290, 529), (33, 70, 2087)])
def test_gemm_long_products(engine, m, n, k, conj_a, conj_b, dtype):
    """K below, at and beyond the line of the longer stages, with remainders of
    a stage and a tile, whole and split K; k eps of the magnitudes."""
    A = _gaussian((k, m + 3) if conj_a else (m, k + 3), dtype, 5)[:, :m if conj_a else k]
    B = _gaussian((n, k + 1) if conj_b else (k, n + 1), dtype, 6)[:, :k if conj_b else n]
    C0 = _gaussian((m, n), dtype, 7)
    C = C0.clone()
    engine.gemm(A, B, C, alpha=0.3, conj_a=conj_a, conj_b=conj_b)
    a, b = A.mH if conj_a else A, B.mH if conj_b else B
    mag = 0.3 * (a.abs() @ b.abs()) + C0.abs()
    assert bool(((C - (C0 + 0.3 * (a @ b))).abs() <= 4 * (k ** 0.5 + 2) * 1.2e-16 * mag).all())


@pytest.mark.parametrize("dtype", _DTYPES)
@pytest.mark.parametrize("n,nrhs", [(1, 8), (31, 3), (64, 8), (65, 1), (127, 5), (128, 8), (129, 8)])
def test_lu_solve_at_the_small_line(engine, n, nrhs, dtype):
    """Substitution for small matrices and the sweep beyond: the solution of a
    dominant system, n eps cond = 129 * 1.1e-16 * ~30 < 1e-12, and the same
    whether the right-hand sides are solved together or alone."""
    hi = torch.complex128 if dtype.is_complex else torch.float64
    LU = (_gaussian((n, n), dtype, n) / n ** 0.5 + 3.0 * torch.eye(n, dtype=dtype, device="cuda")).contiguous()
    piv, _ = engine.lu_factor(LU)
    F = LU.to(hi)
    M = (torch.tril(F, -1) + torch.eye(n, dtype=hi, device="cuda")) @ torch.triu(F)
    b = _gaussian((n, nrhs), hi, 8)
    x = b.clone()
    engine.lu_solve(LU, piv, x)
    pb = b.clone()
    for i, p in enumerate(piv.tolist()):
        pb[[i, p]] = pb[[p, i]]
    ref = torch.linalg.solve(M, pb)
    assert float((x - ref).abs().max()) < 1e-12 * max(1.0, float(ref.abs().max()))
    for c in range(nrhs):
        xc = b[:, c].contiguous()
        engine.lu_solve(LU, piv, xc)
        assert float((xc - x[:, c]).abs().max()) <= 1e-14 * float(x.abs().max())


@pytest.mark.parametrize("cplx", [False, True])
def test_small_solve_with_a_zero_pivot_is_not_finite(engine, cplx):
    """As beyond the line: rows that depend on the zero pivot are infinite or
    NaN, the others are solved."""
    n, z = 90, 70
    dtype = torch.complex128 if cplx else torch.float64
    A = torch.triu(_gaussian((n, n), dtype, 1)) + 9.0 * torch.eye(n, dtype=dtype, device="cuda")
    A[z, z] = 0.0
    b = _gaussian((n, 1), dtype, 2)
    x = b.clone()
    engine.lu_solve(A, torch.arange(n, dtype=torch.int32, device="cuda"), x)
    ref = torch.linalg.solve(A[z + 1:, z + 1:], b[z + 1:])
    assert float((x[z + 1:] - ref).abs().max()) < 1e-12 * float(ref.abs().max())
    x = x.cpu().numpy()
    assert not np.isfinite(x[:z + 1]).any()


def _sphere(engine, sub, Q):
    from bem_b200 import icosphere
    from bem_b200.engine import DeviceSpace
    v, f = icosphere(sub)
    engine.set_mesh(v, f, Q)
    p = np.arange(len(f), dtype=np.int32)
    return v, f, DeviceSpace.from_numpy(p, 1, p, engine.device), DeviceSpace.from_numpy(p, 3, f.reshape(-1).copy(), engine.device)


@pytest.mark.parametrize("cplx", [False, True])
def test_one_point_rule(engine, cplx):
    """GaussQR 1 in FP64: on panels that share no vertex V, K and K' (its second
    block) are the kernels at the rule's points, 1e-13 of the largest entry
    for a dozen roundings and the sine; products against the blocks."""
    from bem_b200 import _lib as L
    v, f, p0, _ = _sphere(engine, 2, 1)
    nt, k = len(f), 2.0 if cplx else 0.0
    dtype = torch.complex128 if cplx else torch.float64
    new = lambda: torch.zeros(nt, nt, dtype=dtype, device="cuda")
    V, K, Kt, KP = new(), new(), new(), new()
    desc = lambda op: engine.op_desc(getattr(L, "OP_" + op), cplx, k, k * k)
    engine.assemble(desc("V"), p0, p0, V)
    engine.assemble(desc("K"), p0, p0, K, 1.0, Kt, -0.5)
    engine.assemble(desc("KP"), p0, p0, KP)
    t = v[f]
    cross = np.cross(t[:, 1] - t[:, 0], t[:, 2] - t[:, 0])
    area2 = np.linalg.norm(cross, axis=1)  # twice the area
    nrm = cross / area2[:, None]
    # the one-point Duffy rule: y = v0 + (v1 - v0) / 2 + (v2 - v1) / 4, weight 1/2
    y = t[:, 0] + 0.5 * (t[:, 1] - t[:, 0]) + 0.25 * (t[:, 2] - t[:, 1])
    d = y[:, None] - y[None]  # x - y
    far = ~np.array([[len(set(a) & set(b)) > 0 for b in f] for a in f])
    r = np.sqrt((d * d).sum(-1)) + ~far
    G = area2[:, None] * area2[None] * 0.25 * (np.exp(1j * k * r) if cplx else 1.0) / (4 * np.pi * r)
    dn = (G * (1 - 1j * k * r if cplx else 1.0) / r ** 2)
    Kref, KPref = dn * np.einsum("ijc,jc->ij", d, nrm), -dn * np.einsum("ijc,ic->ij", d, nrm)
    for got, ref in ((V, G), (K, Kref), (Kt, -0.5 * Kref.T), (KP, KPref)):
        assert np.abs((got.cpu().numpy() - ref)[far]).max() < 1e-13 * np.abs(ref[far]).max()
    x = _gaussian((nt,), dtype, 9)
    for op, A in (("V", V), ("K", K), ("KP", KP)):
        z = torch.zeros(nt, dtype=dtype, device="cuda")
        engine.apply(desc(op), p0, p0, x, z)
        assert float((z - A @ x).abs().max()) < 1e-13 * float((A.abs() @ x.abs()).max())


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("sub,Q", [(0, 3), (2, 3), (3, 2), (4, 1)])
def test_fp64_dirichlet_pass_over_test_panel_counts(engine, sub, Q, cplx):
    """One test panel per CTA, four and eight: the block and the right-hand side
    of the one pass against those of the two calls, both FP64."""
    from bem_b200 import _lib as L
    v, f, p0, p1 = _sphere(engine, sub, Q)
    nt, k = len(f), 2.0 if cplx else 0.0
    dtype = torch.complex128 if cplx else torch.float64
    g = _gaussian((len(v),), dtype, 10)
    A, B = (torch.zeros(nt, nt, dtype=dtype, device="cuda") for _ in range(2))
    a, b = (torch.zeros(nt, dtype=dtype, device="cuda") for _ in range(2))
    engine.assemble_dirichlet(engine.op_desc(L.OP_V, cplx, k, k * k), p0, p0, A, p0, p1, g, a)
    engine.assemble(engine.op_desc(L.OP_V, cplx, k, k * k), p0, p0, B)
    engine.apply(engine.op_desc(L.OP_K, cplx, k, k * k), p0, p1, g, b)
    assert float((A - B).abs().max()) < 1e-13 * float(B.abs().max())
    assert float((a - b).abs().max()) < 1e-12 * float(b.abs().max())


@pytest.mark.parametrize("op", ["V", "K"])
@pytest.mark.parametrize("Q", [1, 2])
def test_shape_adjoint_with_few_points(engine, op, Q):
    """Panels of unequal size, where the vertices' share of a pair outweighs its
    points: central differences of lam . A u, h = 1e-5: truncation h^2 / edge^2
    ~ 1e-8, rounding eps |F| / (h |grad|) ~ 1e-10 of the largest, so 1e-6."""
    from bem_b200 import _lib as L
    v, f, _, _ = _sphere(engine, 1, Q)
    v = v * (1.0 + 0.4 * v[:, :1])
    desc = engine.op_desc(getattr(L, "OP_" + op), False)
    lam, u = (_gaussian((n,), torch.float64, 11) for n in (len(f), len(f) if op == "V" else len(v)))

    def spaces(x):
        from bem_b200.engine import DeviceSpace
        engine.set_mesh(x, f, Q)
        p = np.arange(len(f), dtype=np.int32)
        p0 = DeviceSpace.from_numpy(p, 1, p, engine.device)
        return p0, p0 if op == "V" else DeviceSpace.from_numpy(p, 3, f.reshape(-1).copy(), engine.device)

    def form(x):
        y = torch.zeros(len(f), dtype=torch.float64, device="cuda")
        engine.apply(desc, *spaces(x), u, y)
        return float(lam @ y)

    grad = torch.zeros(len(v), 3, dtype=torch.float64, device="cuda")
    engine.adjoint_vertices(desc, *spaces(v), lam, u, grad)
    grad = grad.cpu().numpy()
    rng = np.random.default_rng(12)
    for _ in range(8):
        d = np.zeros_like(v)
        d[rng.integers(len(v)), rng.integers(3)] = 1e-5
        fd = (form(v + d) - form(v - d)) / 2e-5
        assert abs(fd - (grad * d).sum() / 1e-5) < 1e-6 * np.abs(grad).max()
