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
