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
