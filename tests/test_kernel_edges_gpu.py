"""The kernels at the sizes where their tiles, remainders and dispatch rules
change, against numpy or the CPU oracle."""
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


# ---- the 64 x 64 Cholesky block -------------------------------------------------
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 48, 63, 64, 65, 127, 129])
def test_chol_block_sizes(engine, n, cplx):
    """X = L^-1 of a Hermitian matrix with eigenvalues in about [1, 6]:
    |X N X^H - I| is at most a few n eps cond = 129 * 2.2e-16 * 6 * ~5 = 1e-12;
    L itself to the same."""
    G = _gaussian((2 * n + 8, n), cplx, n)
    N = G.conj().T @ G / (2 * n + 8) + np.eye(n)
    A = torch.as_tensor(N, device="cuda").contiguous()
    X, info = engine.chol_inverse(A)
    assert int(info.item()) == 0
    x = np.tril(X.cpu().numpy())
    low = np.tril(A.cpu().numpy())
    assert np.abs(x @ N @ x.conj().T - np.eye(n)).max() < 1e-12
    assert np.abs(low - np.linalg.cholesky(N)).max() < 1e-12
    assert np.abs(np.triu(X.cpu().numpy(), 1)).max() == 0.0


@pytest.mark.parametrize("col", [0, 16, 63, 64, 100])
def test_chol_block_first_bad_pivot(engine, col):
    """info is 1 + the first column whose pivot is not positive."""
    A = torch.eye(130, dtype=torch.complex128, device="cuda")
    A[col, col] = -1.0
    A[col + 5, col + 5] = float("nan")
    _, info = engine.chol_inverse(A)
    assert int(info.item()) == col + 1


# ---- FP64 separate pairs, one evaluation per unordered pair ------------------------
def _partial_space(f, nv, nb, count, seed):
    """A shuffled part of the panels with a few dofs skipped."""
    rng = np.random.default_rng(seed)
    panels = rng.permutation(len(f))[:count].astype(np.int32)
    dof = panels[:, None].copy() if nb == 1 else f[panels].astype(np.int32).copy()
    dof[rng.random(dof.shape) < 0.03] = -1
    return panels, nb, np.ascontiguousarray(dof.reshape(-1))


@pytest.mark.parametrize("k", [0.0, 0.5, 1.5, 40.0])
@pytest.mark.parametrize("op,nbx,nby", [("V", 1, 1), ("V", 3, 3), ("W", 3, 3), ("K", 1, 3), ("K", 1, 1), ("KP", 3, 1),
                                        ("KP", 1, 1)])
def test_unordered_pairs_over_partial_lists(engine, op, nbx, nby, k):
    """Lists that differ, overlap in part and are in no order: pairs present
    in both orders, in one, and panels absent from either side; the block, its
    transposed copy and the product, in the phase classes (none, <= 0.3,
    <= pi/4, reduced).  1e-12 of the largest entry, as the other FP64 blocks
    (625-term sums in another order)."""
    from bem_b200 import icosphere
    from bem_b200.engine import DeviceSpace
    from oracle import oracle as O
    v, f = icosphere(2)
    engine.set_mesh(v, f, 3)
    code = getattr(O, "OP_" + op)
    helm = k > 0
    ts = _partial_space(f, len(v), nbx, 201, 1)
    rs = _partial_space(f, len(v), nby, 263, 2)
    td, rd = (DeviceSpace.from_numpy(*s, engine.device) for s in (ts, rs))
    n = len(f)
    dt = np.complex128 if helm else np.float64
    ref, ref_t = np.zeros((n, n), dt), np.zeros((n, n), dt)
    O.assemble(v, f, code, helm, k, k * k, 3, True, ts, rs, out=ref, out_t=ref_t, scale=0.7, scale_t=-1.3)
    out, out_t = (torch.zeros(n, n, dtype=torch.complex128 if helm else torch.float64, device="cuda") for _ in "ab")
    desc = engine.op_desc(code, helm, k, k * k)
    engine.assemble(desc, td, rd, out, scale=0.7, out_t=out_t, scale_t=-1.3)
    for got, want in ((out, ref), (out_t, ref_t)):
        assert np.abs(got.cpu().numpy() - want).max() < 1e-12 * np.abs(want).max()
    x = _gaussian(n, helm, 3)
    y = np.zeros(n, dt)
    O.assemble(v, f, code, helm, k, k * k, 3, True, ts, rs, x=x, y=y, scale=-0.5, conj_x=helm)
    yd = torch.zeros(n, dtype=out.dtype, device="cuda")
    engine.apply(desc, td, rd, torch.as_tensor(x, device="cuda"), yd, scale=-0.5, conj_x=helm)
    assert np.abs(yd.cpu().numpy() - y).max() < 1e-12 * np.abs(y).max()


# ---- partial-pivoting LU --------------------------------------------------------------
_EPS = {"float64": 2.3e-16, "complex128": 2.3e-16, "float32": 1.2e-7, "complex64": 1.2e-7}


def _swapped(A, piv):
    A = A.copy()
    for i, p in enumerate(piv):
        A[[i, p]] = A[[p, i]]
    return A


@pytest.mark.parametrize("dtype", list(_EPS))
@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 63, 64, 65, 72, 127, 130, 257, 513, 700, 1089])
def test_lu_panel_sizes(engine, n, dtype):
    """P A = L U with |re| + |im| pivoting (so |l| <= sqrt 2), over the
    cluster sizes of the panel (1 to 16 CTAs), partial panels and partial
    sub-blocks.  |P A - L U| is at most about n eps |L||U| entrywise; a random
    matrix's growth keeps |L||U| below about sqrt(n) max|A| n^(2/3), and
    rounding errors add like sqrt(n): 4 n eps max|U|."""
    cplx = dtype.startswith("complex")
    A = _gaussian((n, n), cplx, n)
    LU = torch.as_tensor(A, device="cuda").to(getattr(torch, dtype)).contiguous()
    A = LU.cpu().numpy().astype(np.complex128 if cplx else np.float64)
    piv, info = engine.lu_factor(LU)
    assert int(info.item()) == 0
    F = LU.cpu().numpy().astype(A.dtype)
    piv = piv.cpu().numpy()
    assert ((piv >= np.arange(n)) & (piv < n)).all()
    low, up = np.tril(F, -1) + np.eye(n), np.triu(F)
    assert np.abs(low).max() <= 1.4143 and np.isfinite(F).all()
    # a lower precision's product of the factors runs on the tensor cores in split TF32
    tol = 4 * max(n, 8) * _EPS[dtype] * np.abs(up).max()
    assert np.abs(_swapped(A, piv) - low @ up).max() < tol


@pytest.mark.parametrize("n,dtype", [(129, "float64"), (1000, "complex128"), (2113, "float64"), (3300, "complex128")])
def test_lu_look_ahead(engine, n, dtype):
    """The next panel beside the update: the same factors every time, bit for
    bit (no race), also where the first panels are too large for a cluster
    (3300 complex rows), and P A = L U as in test_lu_panel_sizes."""
    torch.manual_seed(n)
    A = torch.randn(n, n, dtype=getattr(torch, dtype), device="cuda")
    runs = []
    for _ in range(3):
        LU = A.clone()
        piv, info = engine.lu_factor(LU)
        assert int(info.item()) == 0
        runs.append((LU, piv))
    F, piv = runs[0]
    for LU, p in runs[1:]:
        assert torch.equal(p, piv) and torch.equal(LU, F)
    perm = np.arange(n)
    for i, p in enumerate(piv.cpu().numpy()):
        perm[[i, p]] = perm[[p, i]]
    low, up = torch.tril(F, -1) + torch.eye(n, dtype=F.dtype, device="cuda"), torch.triu(F)
    err = (A[torch.as_tensor(perm, device="cuda")] - low @ up).abs().max()
    assert float(err) < 4 * n * 2.3e-16 * float(up.abs().max())


def test_lu_pivots_match_the_textbook(engine):
    """The pivot sequence of a matrix with ties and exact zeros: the lowest
    row of the largest |re| + |im|."""
    rng = np.random.default_rng(5)
    A = rng.integers(-3, 4, (150, 150)).astype(np.float64)
    ref, want = A.copy(), []
    for j in range(40):  # the steps whose values stay exact enough to tie only where the integers do
        p = j + int(np.argmax(np.abs(ref[j:, j])))
        want.append(p)
        ref[[j, p]] = ref[[p, j]]
        ref[j + 1:, j] /= ref[j, j]
        ref[j + 1:, j + 1:] -= np.outer(ref[j + 1:, j], ref[j, j + 1:])
    piv, _ = engine.lu_factor(torch.as_tensor(A, device="cuda"))
    assert list(piv.cpu().numpy()[:4]) == want[:4]


@pytest.mark.parametrize("col", [0, 5, 70])
def test_lu_zero_and_nan_columns(engine, col):
    """A zero column sets info to 1 + that column; a NaN never becomes a
    pivot while a finite candidate is left."""
    A = np.eye(140) * 3.0
    A[col, col] = 0.0
    _, info = engine.lu_factor(torch.as_tensor(A, device="cuda"))
    assert int(info.item()) == col + 1
    A = np.eye(140) * 3.0
    A[col, col] = np.nan
    A[col + 3, col] = 1.0
    piv, _ = engine.lu_factor(torch.as_tensor(A, device="cuda"))
    assert int(piv[col].item()) == col + 3


# ---- triangular solves ------------------------------------------------------------------
@pytest.mark.parametrize("dtype", ["float64", "complex128", "complex64"])
@pytest.mark.parametrize("n,nrhs", [(1, 1), (63, 2), (64, 1), (65, 3), (129, 8), (200, 1), (1000, 5)])
def test_lu_solve_sizes_and_right_hand_sides(engine, n, nrhs, dtype):
    """x of a well-conditioned system against numpy with the factor as
    stored: n eps cond = 1000 * 2.2e-16 * ~30 < 1e-11 (the solve runs in FP64
    whatever the factor's type, so the comparison takes the factor's own
    product as the matrix)."""
    cplx = dtype.startswith("complex")
    A = _gaussian((n, n), cplx, n) / np.sqrt(n) + 3.0 * np.eye(n)
    LU = torch.as_tensor(A, device="cuda").to(getattr(torch, dtype)).contiguous()
    piv, _ = engine.lu_factor(LU)
    wide = np.complex128 if cplx else np.float64
    F = LU.cpu().numpy().astype(wide)
    M = (np.tril(F, -1) + np.eye(n)) @ np.triu(F)
    B = _gaussian((n, nrhs), cplx, 7)
    x = torch.as_tensor(B, device="cuda")
    engine.lu_solve(LU, piv, x)
    ref = np.linalg.solve(M, _swapped(B, piv.cpu().numpy()))
    assert np.abs(x.cpu().numpy() - ref).max() < 1e-11 * np.abs(ref).max()


@pytest.mark.parametrize("cplx", [False, True])
def test_lu_solve_with_a_zero_pivot_is_not_finite(engine, cplx):
    """A factor with an exact zero on U's diagonal divides by zero: every row
    that depends on it is infinite or NaN, the others are not."""
    n, z = 150, 70
    A = np.triu(_gaussian((n, n), cplx, 1)) + 9.0 * np.eye(n)
    A[z, z] = 0.0
    LU = torch.as_tensor(A, device="cuda")
    piv = torch.arange(n, dtype=torch.int32, device="cuda")
    b = _gaussian((n, 1), cplx, 2)
    x = torch.as_tensor(b, device="cuda")
    engine.lu_solve(LU, piv, x)
    x = x.cpu().numpy()[:, 0]
    ref = np.linalg.solve(A[z + 1:, z + 1:], b[z + 1:, 0])
    assert np.abs(x[z + 1:] - ref).max() < 1e-12 * np.abs(ref).max()
    assert not np.isfinite(x[:z + 1]).any()


# ---- shape adjoint, both orders of a pair from one evaluation ----------------------------
@pytest.mark.parametrize("op,nby", [("V", 1), ("K", 3)])
def test_adjoint_over_partial_lists(engine, op, nby):
    """Lists that differ and overlap in part, zero entries in lam, skipped
    dofs: against central differences (h = 1e-5) of lam . A u.  Truncation
    h^2 / edge^2 ~ 1e-8 and rounding eps |F| / (h |grad|) ~ 1e-10 of the
    largest component; 1e-6 leaves two orders."""
    from bem_b200 import _lib as L
    from bem_b200 import icosphere
    from bem_b200.engine import DeviceSpace
    v, f = icosphere(1)
    ts, rs = _partial_space(f, len(v), 1, 50, 3), _partial_space(f, len(v), nby, 66, 4)
    rng = np.random.default_rng(6)
    lam = rng.standard_normal(len(f))
    lam[::7] = 0.0
    u = rng.standard_normal(len(f) if nby == 1 else len(v))
    lam_d, u_d = torch.as_tensor(lam, device="cuda"), torch.as_tensor(u, device="cuda")
    desc = engine.op_desc(getattr(L, "OP_" + op), False)

    def form(x):
        engine.set_mesh(x, f, 3)
        td, rd = (DeviceSpace.from_numpy(*s, engine.device) for s in (ts, rs))
        y = torch.zeros(len(f), dtype=torch.float64, device="cuda")
        engine.apply(desc, td, rd, u_d, y)
        return float(lam_d @ y), td, rd

    _, td, rd = form(v)
    grad = torch.zeros(len(v), 3, dtype=torch.float64, device="cuda")
    engine.adjoint_vertices(desc, td, rd, lam_d, u_d, grad)
    grad = grad.cpu().numpy()
    for _ in range(12):
        i, c = int(rng.integers(len(v))), int(rng.integers(3))
        h = 1e-5
        p, m = v.copy(), v.copy()
        p[i, c] += h
        m[i, c] -= h
        fd = (form(p)[0] - form(m)[0]) / (2 * h)
        assert abs(fd - grad[i, c]) < 1e-6 * np.abs(grad).max()


@pytest.mark.parametrize("quirk", [True, False])
@pytest.mark.parametrize("Q", [1, 4, 12])
def test_adjoint_data_derivative(engine, Q, quirk):
    """data += K^T lam beside the vertex gradient, over lists that overlap in
    part with skipped dofs and zeros in lam, against the assembled block: the
    same points in another order, sums of at most 162 entries: 1e-12 of the
    largest; the gradient as without it (atomic order: 1e-12)."""
    from bem_b200 import _lib as L
    from bem_b200 import icosphere
    from bem_b200.engine import DeviceSpace
    v, f = icosphere(1)
    v = v * (1.0 + 0.05 * np.sin(3.0 * v[:, :1]))
    engine.set_mesh(v, f, Q)
    td, rd = (DeviceSpace.from_numpy(*_partial_space(f, len(v), nb, c, s), engine.device)
              for nb, c, s in ((1, 50, 3), (3, 66, 4)))
    gen = torch.Generator(device="cuda").manual_seed(8)
    lam = torch.randn(len(f), dtype=torch.float64, device="cuda", generator=gen)
    lam[::7] = 0.0
    u = torch.randn(len(v), dtype=torch.float64, device="cuda", generator=gen)
    u[::5] = 0.0
    desc = engine.op_desc(L.OP_K, False, quirk=quirk)
    K = torch.zeros(len(f), len(v), dtype=torch.float64, device="cuda")
    engine.assemble(desc, td, rd, K)
    grads = [torch.zeros(len(v), 3, dtype=torch.float64, device="cuda") for _ in range(2)]
    data = torch.ones(len(v), dtype=torch.float64, device="cuda")
    engine.adjoint_vertices(desc, td, rd, lam, u, grads[0], data)
    engine.adjoint_vertices(desc, td, rd, lam, u, grads[1])
    ref = 1.0 + (lam[:, None] * K).sum(0)
    assert float((data - ref).abs().max()) < 1e-12 * float(ref.abs().max())
    assert float((grads[0] - grads[1]).abs().max()) < 1e-12 * float(grads[1].abs().max())


@pytest.mark.parametrize("deriv_k", [False, True])
@pytest.mark.parametrize("op", ["V", "W"])
def test_batched_symmetric_blocks_over_partial_lists(engine, op, deriv_k):
    """P1 x P1 blocks of three wavenumbers, lists that overlap in part with
    skipped dofs, a transposed copy: against the one-wavenumber kernel, the
    same FP64 terms in another order (sums of at most ~200): 1e-12."""
    from bem_b200 import _lib as L
    from bem_b200 import icosphere
    from bem_b200.engine import DeviceSpace
    v, f = icosphere(1)
    engine.set_mesh(v, f, 3)
    td, rd = (DeviceSpace.from_numpy(*_partial_space(f, len(v), 3, c, s), engine.device) for c, s in ((50, 3), (66, 4)))
    ks, k2s, scales, scales_t = [0.7, 2.0, 9.0], [0.3, 4.0, 80.0], [1.0, -0.5, 2.0], [0.25, 1.5, -1.0]
    desc = lambda k, k2: engine.op_desc(getattr(L, "OP_" + op), True, k, k2, deriv_k=deriv_k)
    new = lambda: torch.zeros(len(v), len(v), dtype=torch.complex128, device="cuda")
    outs, outs_t = [new() for _ in ks], [new() for _ in ks]
    engine.assemble_batch(desc(0.7, 0.3), td, rd, ks, k2s, outs, scales, outs_t, scales_t)
    for i in range(3):
        ref, ref_t = new(), new()
        engine.assemble(desc(ks[i], k2s[i]), td, rd, ref, scale=scales[i], out_t=ref_t, scale_t=scales_t[i])
        for x, y in ((outs[i], ref), (outs_t[i], ref_t)):
            assert float((x - y).abs().max()) < 1e-12 * float(y.abs().max())


# ---- near pairs ------------------------------------------------------------------------------
@pytest.mark.parametrize("quirk", [True, False])
@pytest.mark.parametrize("Q", [1, 2, 3, 6])
@pytest.mark.parametrize("op,nbx,nby", [("V", 1, 1), ("V", 3, 3), ("K", 1, 3), ("K", 3, 3), ("KP", 3, 1), ("W", 3, 3),
                                        ("W", 1, 1)])
def test_near_pairs_orders_and_batches(engine, op, nbx, nby, Q, quirk):
    """Every point order whose Q^4 points fill part of a warp, a warp, and
    several; one wavenumber and batches of two and three (one launch of two
    and one of one), in each phase class.  On an icosphere of 20 panels most
    pairs touch.  FP64 sums in another order than the oracle's: 1e-12 of the
    largest entry."""
    from bem_b200 import icosphere
    from oracle import oracle as O
    from bem_b200.engine import DeviceSpace
    v, f = icosphere(0)
    engine.set_mesh(v, f, Q)
    code = getattr(O, "OP_" + op)
    full = {1: (np.arange(len(f), dtype=np.int32), 1, np.arange(len(f), dtype=np.int32)),
            3: (np.arange(len(f), dtype=np.int32), 3, f.reshape(-1).copy())}
    ts, rs = full[nbx], full[nby]
    td, rd = (DeviceSpace.from_numpy(*s, engine.device) for s in (ts, rs))
    rows, cols = (len(f) if nb == 1 else len(v) for nb in (nbx, nby))

    def ref(k):
        out = np.zeros((rows, cols), np.complex128)
        O.assemble(v, f, code, True, k, k * k, Q, quirk, ts, rs, out=out)
        return out

    ks = [0.05, 0.25, 3.0]
    want = [ref(k) for k in ks]
    for k, w in zip(ks, want):
        out = torch.zeros(rows, cols, dtype=torch.complex128, device="cuda")
        engine.assemble(engine.op_desc(code, True, k, k * k, quirk=quirk), td, rd, out)
        assert np.abs(out.cpu().numpy() - w).max() < 1e-12 * np.abs(w).max()
    for count in (2, 3):
        outs = [torch.zeros(rows, cols, dtype=torch.complex128, device="cuda") for _ in range(count)]
        engine.assemble_batch(engine.op_desc(code, True, quirk=quirk), td, rd, ks[:count], [k * k for k in ks[:count]],
                              outs, [1.0] * count)
        for o, w in zip(outs, want):
            assert np.abs(o.cpu().numpy() - w).max() < 1e-12 * np.abs(w).max()


# ---- tile-pivoted LU -------------------------------------------------------------------------
@pytest.mark.parametrize("dtype", ["float32", "complex64", "float64", "complex128"])
@pytest.mark.parametrize("n", [1, 15, 16, 17, 63, 64, 65, 100, 128, 191, 330])
def test_tile_lu_sizes(engine, n, dtype):
    """P A = L U with row swaps inside each 64-row tile, |l| <= sqrt 2 inside
    the diagonal tiles, and the tile's first pivot the largest |re| + |im| of
    its first column.  A diagonally dominant random matrix keeps the factors
    of the size of A: n eps max|A|, times 8 for the split TF32 products."""
    cplx = dtype.startswith("complex")
    A = _gaussian((n, n), cplx, n + 1) / np.sqrt(n) + 2.0 * np.eye(n)
    LU = torch.as_tensor(A, device="cuda").to(getattr(torch, dtype)).contiguous()
    A = LU.cpu().numpy().astype(np.complex128 if cplx else np.float64)
    piv, _, info = engine.lu_factor_tiled(LU)
    assert int(info.item()) == 0
    F = LU.cpu().numpy().astype(A.dtype)
    piv = piv.cpu().numpy()
    tile = np.arange(n) // 64 * 64
    assert ((piv >= np.arange(n)) & (piv < np.minimum(tile + 64, n))).all()
    first = A[:64, 0]
    assert piv[0] == int(np.argmax(np.abs(first.real) + np.abs(first.imag)))
    low, up = np.tril(F, -1) + np.eye(n), np.triu(F)
    for t in range(0, n, 64):
        assert np.abs(low[t:t + 64, t:t + 64]).max() <= 1.4143
    assert np.abs(_swapped(A, piv) - low @ up).max() < 8 * max(n, 16) * _EPS[dtype] * np.abs(A).max()


@pytest.mark.parametrize("col", [0, 20, 63, 64, 90])
def test_tile_lu_zero_and_nan_columns(engine, col):
    A = torch.eye(100, dtype=torch.float32, device="cuda") * 2.0
    A[col, col] = 0.0
    _, _, info = engine.lu_factor_tiled(A)
    assert int(info.item()) == col + 1
    if col % 64 < 60 and col + 3 < 100:
        A = torch.eye(100, dtype=torch.float32, device="cuda") * 2.0
        A[col, col] = float("nan")
        A[col + 3, col] = 1.0
        piv, _, _ = engine.lu_factor_tiled(A)
        assert int(piv[col].item()) == col + 3


# ---- FP64 tensor-core products --------------------------------------------------------------
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("conj_a,conj_b", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (63, 65, 7), (64, 64, 8), (130, 66, 33), (65, 129, 200), (70, 70, 1100),
                                   (830, 770, 20)])
def test_gemm_edges(engine, m, n, k, conj_a, conj_b, cplx):
    """C += alpha op(A) op(B) with leading dimensions beyond the widths, tiles
    and stages partly filled, fewer stages than the ring, split K (k = 1100),
    tiles of 32 rows and (more tiles than SMs) of 64: k eps max|A| max|B| sqrt-ish sums, 1e-13 k of the result."""
    dt = torch.complex128 if cplx else torch.float64

    def padded(r, c, seed):
        return torch.as_tensor(_gaussian((r, c + 3), cplx, seed), device="cuda", dtype=dt)[:, :c]

    A, B, C = padded(*((k, m) if conj_a else (m, k)), 1), padded(*((n, k) if conj_b else (k, n)), 2), padded(m, n, 3)
    opA, opB = (X.conj().T if c else X for X, c in ((A, conj_a), (B, conj_b)))
    want = (C + 0.75 * opA @ opB).cpu().numpy()
    engine.gemm(A, B, C, alpha=0.75, conj_a=conj_a, conj_b=conj_b)
    assert np.abs(C.cpu().numpy() - want).max() < 1e-13 * max(k, 8) ** 0.5 * 10


def test_gemm_on_unaligned_complex_operands(engine):
    """Complex operands that start on an odd multiple of 8 bytes take 8-byte
    copies."""
    n = 70
    raw = torch.zeros(2 * n * n + 1, dtype=torch.float64, device="cuda")
    raw[1:] = torch.as_tensor(_gaussian((2 * n * n,), False, 4), device="cuda")
    A = torch.as_tensor(_gaussian((n, n), True, 5), device="cuda")
    C = torch.zeros(n, n, dtype=torch.complex128, device="cuda")
    L = engine.lib
    import ctypes
    from bem_b200 import _lib
    rc = L.bem_gemm(engine.ctx, _lib.C128, 0, 0, 0, n, n, n, 1.0, ctypes.c_void_p(raw.data_ptr() + 8), n,
                    ctypes.c_void_p(A.data_ptr()), n, ctypes.c_void_p(C.data_ptr()), n,
                    ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    B = raw[1:].cpu().numpy().reshape(n, n, 2)
    want = (B[..., 0] + 1j * B[..., 1]) @ A.cpu().numpy()
    assert np.abs(C.cpu().numpy() - want).max() < 1e-12 * 10


def test_lu_of_an_unaligned_complex_matrix(engine):
    """A complex128 matrix that starts on an odd multiple of 8 bytes is read
    half an element at a time: the same pivots, and the same factors to
    rounding (n eps)."""
    import ctypes
    from bem_b200 import _lib
    n = 129
    A = torch.as_tensor(_gaussian((n, n), True, 9), device="cuda")
    raw = torch.zeros(2 * n * n + 1, dtype=torch.float64, device="cuda")
    raw[1:] = torch.view_as_real(A).reshape(-1)
    piv2 = torch.empty(n, dtype=torch.int32, device="cuda")
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    rc = engine.lib.bem_lu_factor(engine.ctx, _lib.C128, ctypes.c_void_p(raw.data_ptr() + 8), n, n,
                                  ctypes.c_void_p(piv2.data_ptr()), ctypes.c_void_p(info.data_ptr()),
                                  ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0 and int(info.item()) == 0
    piv, _ = engine.lu_factor(A)
    assert torch.equal(piv, piv2)
    assert float((raw[1:] - torch.view_as_real(A).reshape(-1)).abs().max()) < n * 2.3e-16 * float(A.abs().max())


# ---- products with dense matrices ------------------------------------------------------
@pytest.mark.parametrize("dtype", ["float64", "complex128", "float32", "complex64"])
@pytest.mark.parametrize("m,n", [(1, 1), (9, 31), (8, 128), (65, 129), (70, 256), (3, 517)])
def test_gemv_remainders(engine, m, n, dtype):
    """Around the unrolled part of a row (4 or 8 x 32 elements), rows further
    apart than they are long, complex data at odd multiples of 8 bytes: FP64
    sums of n terms, n eps times the sum of magnitudes."""
    import ctypes
    cplx = dtype.startswith("complex")
    A = torch.as_tensor(_gaussian((m, n + 3), cplx, n), device="cuda").to(getattr(torch, dtype))[:, :n]
    x = _gaussian(n, cplx, m + n)
    y0 = _gaussian(m, cplx, 3)
    a = A.cpu().numpy().astype(x.dtype)
    bound = 2 * (n + 4) * 2.3e-16 * (np.abs(a) @ np.abs(x) + np.abs(y0)).max()
    want = 0.5 * y0 - 2.0 * a @ x
    y = torch.as_tensor(y0.copy(), device="cuda")
    engine.gemv(A, torch.as_tensor(x, device="cuda"), y, alpha=-2.0, beta=0.5)
    assert np.abs(y.cpu().numpy() - want).max() <= bound
    if dtype == "complex128":
        raw = torch.zeros(2 * n + 1, dtype=torch.float64, device="cuda")
        raw[1:] = torch.view_as_real(torch.as_tensor(x, device="cuda")).reshape(-1)
        y = torch.as_tensor(y0.copy(), device="cuda")
        rc = engine.lib.bem_gemv(engine.ctx, 1, ctypes.c_void_p(A.data_ptr()), m, n, A.stride(0),
                                 ctypes.c_void_p(raw.data_ptr() + 8), ctypes.c_void_p(y.data_ptr()), -2.0, 0.5,
                                 ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == 0 and np.abs(y.cpu().numpy() - want).max() <= bound


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("n", [1, 3, 31, 33, 100, 257])
def test_lstsq_products_remainders(engine, n, cplx):
    """min |[A; P] x - b| at sizes around the row chunks of the adjoint
    product (32 rows, 4 at a time): A and P well conditioned (3 I + noise of
    norm about 1), so the refined solution is the least squares one to about
    1e-10."""
    A, P = (3.0 * np.eye(n) + _gaussian((n, n), cplx, n + i) / (3 * np.sqrt(n)) for i in (1, 2))
    b = _gaussian(2 * n, cplx, 7)
    A_, P_ = (torch.as_tensor(M, device="cuda").to(torch.complex128 if cplx else torch.float64) for M in (A, P))
    N = torch.empty_like(A_)
    d = torch.empty(n, dtype=torch.float64, device="cuda")
    engine.gram(A_, P_, N, d, tensor_cores=False)
    piv, dinv, _ = engine.chol_factor(N, tensor_cores=False)
    x = torch.zeros(n, dtype=A_.dtype, device="cuda")
    engine.lstsq_refine(A_, P_, d, N, piv, dinv, torch.as_tensor(b, device="cuda").to(A_.dtype), x)
    want = np.linalg.lstsq(np.vstack([A, P]), b, rcond=None)[0]
    assert np.abs(x.cpu().numpy() - want).max() < 1e-10 * max(1.0, np.abs(want).max())


# ---- both wavenumbers of the Calderon sweep over lane pairs ---------------------------
@pytest.mark.parametrize("ks", [(0.1, 0.05), (1.2, 0.4), (30.0, 45.0), (0.7, -0.3)])
@pytest.mark.parametrize("Q", [1, 2, 3])
def test_calderon_lane_pairs(engine, ks, Q):
    """Odd and even numbers of points and the phase classes (<= 0.3, <= pi/4,
    reduced), over a part of the panels in no order.  FP64 against one
    launch per wavenumber, sums in another order: 1e-12 of the largest entry;
    mixed: the same FP32 values and sums, the FP64 ones in another order
    (atomics): 1e-12 too."""
    from bem_b200 import _lib as L
    from bem_b200 import icosphere
    from bem_b200.engine import DeviceSpace
    from oracle import oracle as O
    v, f = icosphere(2)
    engine.set_mesh(v, f, Q)
    panels, _, dof = _partial_space(f, len(v), 1, 233, 5)
    dof3 = f[panels].astype(np.int32)
    dof3[np.random.default_rng(6).random(dof3.shape) < 0.03] = -1
    dof3[dof3 >= 0] += len(f)
    n = len(f) + len(v)
    neu = DeviceSpace.from_numpy(panels, 1, dof, engine.device)
    dirs = DeviceSpace.from_numpy(panels, 3, np.ascontiguousarray(dof3.reshape(-1)), engine.device)
    for prec in (L.PREC_FP64, L.PREC_MIXED):
        desc = engine.op_desc(O.OP_V, True, ks[0], ks[0] ** 2, precision=prec)
        got = []
        for form in (1, 0):
            engine.set_tuning(L.TUNE_CALDERON_GROUP, form)
            outs = [torch.zeros(n, n, dtype=torch.complex128, device="cuda") for _ in ks]
            engine.assemble_calderon(desc, ks, [k * k for k in ks], neu, dirs, outs, (-1.0, 0.7))
            got.append(outs)
        engine.set_tuning(L.TUNE_CALDERON_GROUP, 0)
        for want, out in zip(*got):
            assert float(want.abs().max()) > 0
            assert float((want - out).abs().max()) < 1e-12 * float(want.abs().max())
