"""The dense solvers and kernels at the ends of the number range and at the
last digits, against extended precision (numpy's long double) or CUDA."""
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


def _gaussian(shape, cplx, seed):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal(shape)
    return x + 1j * rng.standard_normal(shape) if cplx else x


def _gepp(A):
    """L U of A with its rows swapped, in A's own type; the permuted A is not kept."""
    A = A.copy()
    for j in range(len(A)):
        p = j + int(np.argmax(np.abs(A[j:, j])))
        A[[j, p]] = A[[p, j]]
        A[j + 1:, j] /= A[j, j]
        A[j + 1:, j + 1:] -= np.outer(A[j + 1:, j], A[j, j + 1:])
    return A


def _backward_error(F, x, b):
    """Componentwise: max |L U x - b| / (|L||U||x| + |b|), in long double."""
    wide = np.clongdouble if np.iscomplexobj(F) else np.longdouble
    F, x, b = F.astype(wide), x.astype(wide), b.astype(wide)
    low, up = np.tril(F, -1) + np.eye(len(F)), np.triu(F)
    res = np.abs(low @ (up @ x) - b)
    return float((res / (np.abs(low) @ (np.abs(up) @ np.abs(x)) + np.abs(b))).max())


def _solve(engine, F, b):
    n = len(F)
    piv = torch.arange(n, dtype=torch.int32, device="cuda")
    x = torch.as_tensor(b, device="cuda").clone()
    engine.lu_solve(torch.as_tensor(F, device="cuda"), piv, x)
    return x.cpu().numpy()


@pytest.mark.parametrize("dtype", ["float32", "complex64", "float64", "complex128"])
@pytest.mark.parametrize("n", [64, 200])
def test_lu_solve_is_backward_stable(engine, n, dtype):
    """The factors of a Gaussian matrix (not dominant), solved in FP64 whatever
    their type: two triangles of n products, sqrt(n) roundings of 1.1e-16 each
    against the sum of their magnitudes (substitution in numpy: 2e-17 to 6e-17)."""
    F = _gepp(_gaussian((n, n), dtype.startswith("complex"), n).astype(dtype))
    b = _gaussian((n, 3), dtype.startswith("complex"), 1)
    x = _solve(engine, F, b)
    assert _backward_error(F, x, b) < np.sqrt(n) * 1.2e-16


@pytest.mark.parametrize("dtype,exp", [("float32", -80), ("float32", -100), ("float32", 66), ("complex64", -80),
                                       ("complex64", 66), ("float64", -550), ("float64", 520), ("complex128", -550),
                                       ("complex128", 520)])
def test_lu_solve_where_squares_leave_the_range(engine, dtype, exp):
    """U scaled by 2^exp: the pivots are ordinary numbers of their type, their
    squares are not.  Bound as above."""
    n = 130
    F = _gepp(_gaussian((n, n), dtype.startswith("complex"), 3).astype(dtype))
    F = (np.tril(F, -1) + np.triu(F) * np.ldexp(1.0, exp).astype(F.real.dtype)).astype(dtype)
    b = _gaussian((n, 2), dtype.startswith("complex"), 4)
    x = _solve(engine, F, b)
    assert np.isfinite(x).all()
    assert _backward_error(F, x, b) < np.sqrt(n) * 1.2e-16


@pytest.mark.parametrize("dtype", ["float32", "complex64", "float64", "complex128"])
def test_lu_solve_where_a_tile_inverse_overflows(engine, dtype):
    """U = I - 2^20 (superdiagonal), x of small integers: the inverse holds
    2^1260, substitution has integers only and is exact."""
    n = 100
    F = (np.eye(n) - 2.0 ** 20 * np.eye(n, k=1)).astype(dtype)
    cplx = dtype.startswith("complex")
    if cplx:
        F = (F.astype(np.complex128) * (1 + 1j)).astype(dtype)
    F = np.triu(F)
    x0 = np.rint(4 * _gaussian((n, 2), cplx, 5))
    b = F.astype(np.complex128 if cplx else np.float64) @ x0
    assert np.array_equal(_solve(engine, F, b), x0)


# ---- zero pivots by rounding -------------------------------------------------------------
@pytest.fixture(scope="module")
def manager():
    from bem_b200.managers import CoreManager
    from tests._util import load_fixture, torch_callbacks
    d = load_fixture("cube_lap_neu_q5")
    params = eval(str(d["params"]))
    params.update(vertices=d["vertices"], panels=d["panels"])
    core = CoreManager(params)
    core.initialization(*torch_callbacks(str(d["data_kind"]), float(params.get("k", 0.0)), d["direction"]))
    yield core._BEM_manager
    core.kill()


def test_a_pivot_that_rounds_to_zero_does_not_raise(manager):
    """[[3, 1], [1, fl(1/3)]] is not singular (determinant -2^-54), but its
    second pivot is fl(1/3) - fl(1/3) = 0; the other way round it is 1 - 3
    fl(1/3) = 2^-54 in one FMA.  The solution's residual is a few roundings of
    |A||x|; a matrix with a zero column raises."""
    A = np.array([[3.0, 1.0], [1.0, 1.0 / 3.0]])
    b = _gaussian((2, 2), False, 1)
    Ad, bd = torch.as_tensor(A, device="cuda"), torch.as_tensor(b, device="cuda")
    assert int(manager.engine.lu_factor(Ad.clone())[1].item()) == 2
    x = manager._lu_solve_fp64(Ad, bd, [bd[:, 0].contiguous(), bd[:, 1].contiguous()]).cpu().numpy()
    res = np.abs(A.astype(np.longdouble) @ x.astype(np.longdouble) - b)
    assert (res <= 4 * 2.3e-16 * (np.abs(A) @ np.abs(x) + np.abs(b))).all()
    Ad[:, 1] = 0.0
    with pytest.raises(torch.linalg.LinAlgError, match="singular"):
        manager._lu_solve_fp64(Ad, bd[:, 0], [bd[:, 0].contiguous()])


def test_laplace_neumann_never_raises(manager):
    """The pure Neumann cube: 500 assemblies, each its own order of the atomic
    sums, are all solved."""
    for _ in range(500):
        manager._mat_A.zero_()
        manager.run()


# ---- pivots whose square leaves the range --------------------------------------------------
@pytest.mark.parametrize("dtype,exp,tiled", [
    (t, e, tiled)
    for t, e in [("float32", -80), ("float32", 66), ("complex64", -66), ("complex64", -80), ("complex64", 66),
                 ("float64", -550), ("float64", 520), ("complex128", -515), ("complex128", -550), ("complex128", 520)]
    for tiled in (False, True)
    if not (tiled and t in ("float64", "complex128"))])  # the tile factor compares its candidates in FP32
def test_lu_is_equivariant_under_powers_of_two(engine, dtype, exp, tiled):
    """2^exp A has A's pivots and L, and 2^exp U: all operations but the
    products that test the pivots' size scale exactly.  FP32 factors above one
    tile would also use the tensor cores' split, so one tile is taken; rounding
    of the reciprocal alone may differ (1/a from |a|^2 or from the scaled a),
    a few eps of a Gaussian factor's growth, 64 eps max|F|."""
    n = 64
    A = _gaussian((n, n), dtype.startswith("complex"), 9).astype(dtype)
    A += 4 * np.eye(n, dtype=dtype)
    scale = np.ldexp(1.0, exp)
    out = []
    for f in (1.0, scale):
        LU = torch.as_tensor(A * np.asarray(f, A.real.dtype), device="cuda").contiguous()
        piv, *_, info = (engine.lu_factor_tiled if tiled else engine.lu_factor)(LU)
        assert int(info.item()) == 0
        F = LU.cpu().numpy().astype(np.clongdouble if np.iscomplexobj(A) else np.longdouble)
        out.append((piv.cpu().numpy(), np.tril(F, -1) + np.triu(F) / f))
    (p0, F0), (p1, F1) = out
    assert np.array_equal(p0, p1)
    eps = 2.3e-16 if dtype in ("float64", "complex128") else 1.2e-7
    assert np.abs(F1 - F0).max() < 64 * eps * np.abs(F0).max()


# ---- FP64 root and phase of the quadrature kernels ----------------------------------------
def _device_math(engine, which, x):
    x = torch.as_tensor(np.ascontiguousarray(x), device="cuda")
    a, b = torch.empty_like(x), torch.empty_like(x)
    engine._check(engine.lib.bem_device_math(engine.ctx, which, x.data_ptr(), a.data_ptr(), b.data_ptr(), x.numel(),
                                             torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    return x, a.cpu().numpy(), b.cpu().numpy()


def test_root_and_reciprocal_root_to_the_last_digit(engine):
    """sqrt x and 1/sqrt x within 1 ulp (half an ulp for the last rounding,
    half for that of p = x y), over the whole range of normal numbers and
    densely around powers of two; within one more of CUDA's; the ends."""
    rng = np.random.default_rng(1)
    m = np.concatenate([rng.uniform(1.0, 4.0, 400000), 1.0 + np.arange(64) * 2.0 ** -52, 4.0 - np.arange(1, 65) * 2.0 ** -51])
    x = np.concatenate([m, np.ldexp(m, 2 * rng.integers(-510, 511, len(m)))])
    x = x[(x >= 2.3e-308) & np.isfinite(x)]
    xd, r, rinv = _device_math(engine, 0, x)
    root = np.sqrt(x.astype(np.longdouble))
    assert (np.abs(r - root) <= 1.01 * np.spacing(r)).all()
    assert (np.abs(rinv - 1 / root) <= 1.01 * np.spacing(rinv)).all()
    assert (np.abs(rinv - torch.rsqrt(xd).cpu().numpy()) <= 2 * np.spacing(rinv)).all()
    _, _, rinv = _device_math(engine, 0, np.array([0.0, np.inf, np.nan, -1.0]))
    assert rinv[0] == np.inf and rinv[1] == 0.0 and np.isnan(rinv[2:]).all()


@pytest.mark.parametrize("which,bound", [(2, np.pi / 4), (3, 0.3)])
def test_short_sine_and_cosine(engine, which, bound):
    """Half an ulp for the last rounding, half for the first dropped term, the
    rest of Horner's scheme enters with y^2 / 2: 1.5 ulp."""
    rng = np.random.default_rng(2)
    x = np.concatenate([rng.uniform(-bound, bound, 400000), bound * 2.0 ** -rng.uniform(0, 60, 100000), [0.0, bound]])
    xd, s, c = _device_math(engine, which, x)
    wide = x.astype(np.longdouble)
    assert (np.abs(s - np.sin(wide)) <= 1.5 * np.spacing(np.abs(s))).all()
    assert (np.abs(c - np.cos(wide)) <= 1.5 * np.spacing(c)).all()


def test_sine_and_cosine_of_any_phase(engine):
    """2.3e-16 absolute (two roundings of the reduced argument, one ulp of the
    polynomials) up to the switch at 1e5, next to multiples of pi/2 and on
    both sides of the switch; beyond it CUDA's own; infinities and NaN."""
    rng = np.random.default_rng(3)
    near = np.rint(rng.uniform(0, 63661, 100000)) * (np.pi / 2)
    near = np.nextafter(near, near * (1 + rng.choice([-1, 1], len(near)) * 1e-3))
    x = np.concatenate([rng.uniform(-1e5, 1e5, 400000), rng.uniform(-7, 7, 100000), near, 10.0 ** rng.uniform(-300, 5, 50000),
                        1e5 + np.arange(-64, 65) * np.spacing(1e5), [0.0]])
    xd, s, c = _device_math(engine, 1, x)
    wide = x.astype(np.longdouble)
    assert np.abs(s - np.sin(wide)).max() < 2.3e-16 and np.abs(c - np.cos(wide)).max() < 2.3e-16
    assert np.abs(s - torch.sin(xd).cpu().numpy()).max() < 4.6e-16
    assert np.abs(c - torch.cos(xd).cpu().numpy()).max() < 4.6e-16
    x = np.concatenate([rng.uniform(1e5, 1e9, 1000), 2.0 ** rng.uniform(17, 1000, 1000)])
    xd, s, c = _device_math(engine, 1, x)
    assert np.abs(s - torch.sin(xd).cpu().numpy()).max() < 2.3e-16
    _, s, c = _device_math(engine, 1, np.array([np.inf, -np.inf, np.nan]))
    assert np.isnan(s).all() and np.isnan(c).all()


# ---- negative wavenumbers ------------------------------------------------------------------
def _spaces(engine, v, f):
    from bem_b200.engine import DeviceSpace
    p = np.arange(len(f), dtype=np.int32)
    return (DeviceSpace.from_numpy(p, 1, p, engine.device), DeviceSpace.from_numpy(p, 3, f.reshape(-1).copy(), engine.device))


@pytest.mark.parametrize("k", [-40.0, -0.2])
def test_mixed_precision_at_negative_wavenumbers(engine, k):
    """Blocks, products and the Dirichlet pass against FP64: the FP32 phase k (r
    - R), up to 40 * 2 * 0.35 = 28, carries 6e-8 of itself: 28 * 6e-8 =
    1.7e-6 of an entry, 5e-6 of the largest."""
    from bem_b200 import _lib as L
    from bem_b200 import icosphere
    v, f = icosphere(1)
    engine.set_mesh(v, f, 3)
    p0, p1 = _spaces(engine, v, f)
    g = torch.as_tensor(_gaussian(len(v), True, 6), device="cuda")
    x0 = torch.as_tensor(_gaussian(len(f), True, 7), device="cuda")
    res = []
    for prec in (L.PREC_FP64, L.PREC_MIXED):
        new = lambda *s: torch.zeros(*s, dtype=torch.complex128, device="cuda")
        out = []
        for op, t, r in ((L.OP_V, p0, p0), (L.OP_K, p0, p1), (L.OP_KP, p1, p0), (L.OP_W, p1, p1)):
            nt, nr = (len(f) if s is p0 else len(v) for s in (t, r))
            desc = engine.op_desc(op, True, k, k * k, precision=prec)
            out.append(new(nt, nr))
            engine.assemble(desc, t, r, out[-1])
            out.append(new(nt))
            engine.apply(desc, t, r, x0 if r is p0 else g, out[-1])
        out += [new(len(f), len(f)), new(len(f))]
        engine.assemble_dirichlet(engine.op_desc(L.OP_V, True, k, k * k, precision=prec), p0, p0, out[-2], p0, p1, g, out[-1])
        res.append(out)
    for want, got in zip(*res):
        assert float((got - want).abs().max()) < 5e-6 * float(want.abs().max())


# ---- lists that name a panel twice -----------------------------------------------------------
@pytest.mark.parametrize("op,nbx,nby", [("V", 3, 3), ("W", 3, 3), ("K", 1, 3), ("KP", 3, 1)])
def test_panels_named_twice(engine, op, nbx, nby):
    """Separate pairs count once per entry of either list, touching ones once
    per panel: against the sum of calls without repeats, at FP64's last digits
    (sums of up to ~300 terms in another order: 1e-12 of the largest)."""
    from bem_b200 import _lib as L
    from bem_b200 import icosphere
    from bem_b200.engine import DeviceSpace
    v, f = icosphere(1)
    engine.set_mesh(v, f, 3)
    touch = (f[:, None, :, None] == f[None, :, None, :]).any((2, 3))
    rng = np.random.default_rng(11)
    ts, rs = rng.permutation(len(f))[:50], rng.permutation(len(f))[:60]
    te = rng.choice(np.intersect1d(ts, rs), 6, replace=False)
    re = rng.choice(np.intersect1d(ts, rs), 5, replace=False)

    def space(p, nb):  # as a C caller can pass it; from_numpy refuses repeats
        p = torch.as_tensor(np.asarray(p, np.int32), device="cuda")
        dof = p if nb == 1 else torch.as_tensor(f.astype(np.int32), device="cuda")[p.long()].reshape(-1).contiguous()
        return DeviceSpace(p, nb, dof)

    rows, cols = (len(f) if nb == 1 else len(v) for nb in (nbx, nby))
    desc = engine.op_desc(getattr(L, "OP_" + op), False)
    x = torch.as_tensor(_gaussian(cols, False, 12), device="cuda")
    lam = torch.as_tensor(_gaussian(rows, False, 13), device="cuda")

    def call(t, r, acc):
        td, rd = space(t, nbx), space(r, nby)
        engine.assemble(desc, td, rd, acc[0])
        engine.apply(desc, td, rd, x, acc[1])
        if op == "K":
            engine.adjoint_vertices(desc, td, rd, lam, x, acc[2], acc[3])

    new = lambda: [torch.zeros(s, dtype=torch.float64, device="cuda") for s in ((rows, cols), (rows,), (len(v), 3), (cols,))]
    want, got = new(), new()
    call(ts, rs, want)
    for e in te:
        call([e], rs[~touch[e, rs]], want)
        for g in re[~touch[e, re]]:
            call([e], [g], want)
    for g in re:
        call(ts[~touch[ts, g]], [g], want)
    call(np.concatenate([ts, te]), np.concatenate([rs, re]), got)
    for w, g in zip(want, got):
        assert float((w - g).abs().max()) <= 1e-12 * float(w.abs().max())


def test_solve_with_any_bits_in_the_right_hand_side(engine):
    """A right-hand side that holds the very NaN that marks an unwritten value
    of the sweep is a NaN like any other: no wait runs out."""
    n = 200
    b = torch.ones(n, dtype=torch.float64, device="cuda")
    b.view(torch.int64)[70] = 0x7FF4DEADBEEF0001
    F = torch.eye(n, dtype=torch.float64, device="cuda")
    piv = torch.arange(n, dtype=torch.int32, device="cuda")
    x = b.clone()
    engine.lu_solve(F, piv, x)
    assert bool(x[70].isnan())
    LU = torch.eye(n, dtype=torch.float32, device="cuda")
    tpiv, dinv, _ = engine.lu_factor_tiled(LU)
    y = b.clone()
    engine.lu_solve_tiled(LU, tpiv, dinv, y)
    assert bool(y[70].isnan())


# ---- pivot sequence --------------------------------------------------------------------------
def _exact_elimination(n, cplx, seed):
    """Rows in random order of L U with L in {0, 1/2 (unit)} and U of integers
    with powers of two (times a unit) on its diagonal, and n / 4 planted ties: a
    row r that repeats the pivot row j up to column j (times a unit) has |l| = 1
    there, and whichever of the two becomes the pivot, the other goes on as row r.
    Every value of the elimination is a small dyadic number."""
    rng = np.random.default_rng(seed)
    units = np.array([1, -1, 1j, -1j]) if cplx else np.array([1.0, -1.0])
    pick = lambda *s: units[rng.integers(0, len(units), s)]
    low = np.tril(0.5 * pick(n, n) * (rng.random((n, n)) < 0.5), -1)
    up = np.triu(rng.integers(-3, 4, (n, n)) * pick(n, n), 1) + np.diag(2.0 ** rng.integers(0, 3, n) * pick(n))
    pairs = np.sort(rng.permutation(n)[:n // 4 * 2].reshape(-1, 2), 1)
    low[:, pairs[:, 0]] = 0.0
    for j, r in pairs:
        s = pick(1)[0]
        low[r, :j] = s * low[j, :j]
        low[r, j] = s
    return ((low + np.eye(n)) @ up)[rng.permutation(n)]


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("n", [40, 150, 700])
def test_every_pivot_matches_the_textbook(engine, n, cplx):
    """The whole pivot sequence, ties included (the lowest row of the largest
    |re| + |im|), over several sub-blocks, panels and CTAs: exact arithmetic,
    so the sequence and the factors are equal."""
    A = _exact_elimination(n, cplx, n)
    assert np.array_equal(A * 2, np.rint(A.real * 2) + (1j * np.rint(A.imag * 2) if cplx else 0.0))
    ref, want, ties = A.copy(), [], 0
    for j in range(n):
        size = np.abs(ref[j:, j].real) + np.abs(ref[j:, j].imag)
        p = j + int(np.argmax(size))
        ties += int((size == size.max()).sum() > 1)
        want.append(p)
        ref[[j, p]] = ref[[p, j]]
        ref[j + 1:, j] *= 1.0 / ref[j, j]
        ref[j + 1:, j + 1:] -= np.outer(ref[j + 1:, j], ref[j, j + 1:])
    assert ties >= n // 8
    LU = torch.as_tensor(A, device="cuda")
    piv, info = engine.lu_factor(LU)
    assert int(info.item()) == 0
    assert list(piv.cpu().numpy()) == want
    assert np.array_equal(LU.cpu().numpy(), ref)
