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
