"""The tcgen05 products (7 base-256 digits, two halves of 32 columns a tile) against NumPy: lengths around a k-step, a
fold interval (160) and several of them, rows and columns around the tiles, real and complex, beta, the paired form."""

import numpy as np
import pytest

from taurus_vap_gb300 import model as M
from taurus_vap_gb300.native import Context

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    return Context(M.sd_model(seed=2).basis)


# at least 152 tiles of 128 x 64 (of the doubled rows of a complex operand), and more than 1.2e7 multiply-adds
@pytest.mark.parametrize("m,n,k", [(2433, 513, 16), (2560, 480, 17), (2433, 545, 159), (2561, 512, 160),
                                   (1300, 1000, 161), (2560, 491, 320), (4100, 300, 337), (2433, 577, 1000)])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("halves", [1, 2])
def test_tcgen05_products(ctx, m, n, k, cplx, halves):
    rng = np.random.default_rng(k + 13 * m)

    def mat(r, c):
        x = rng.normal(size=(r, c)) * 10.0 ** rng.integers(-8, 9, size=(r, 1))
        return x + 1j * rng.normal(size=(r, c)) * 10.0 ** rng.integers(-8, 9, size=(r, 1)) if cplx else x

    A, B = mat(m, k), mat(n, k).T  # rows of op(A) and columns of op(B) of very different sizes
    C = mat(m, n)
    ref = A @ B
    big = lambda x, ax: np.maximum(np.abs(x.real), np.abs(x.imag)).max(axis=ax)  # noqa: E731
    # the documented bound, and the rounding of NumPy's own sum of K terms
    bound = (2.0 ** -46 if cplx else 2.0 ** -49) * k * np.outer(big(A, 1), big(B, 0)) + \
        4 * k * 2.0 ** -53 * (np.abs(A) @ np.abs(B))
    ctx.set_tuning(0 if halves == 2 else 2, 2, 0)
    got = ctx.gemm(A, B)
    assert np.all(np.abs(got - ref) <= bound)
    got = ctx.gemm(A, B, beta=-0.5, C=C)
    assert np.all(np.abs(got - (ref - 0.5 * C)) <= bound + 2.0 ** -50 * (np.abs(ref) + np.abs(C)))
    if cplx:
        ctx.set_option(ctx.OPT_COMPLEX_PAIRS, 1)
        pairs = ctx.gemm(A, B)
        ctx.set_option(ctx.OPT_COMPLEX_PAIRS, 0)
        assert np.array_equal(pairs, ctx.gemm(A, B))
    ctx.set_tuning(0, 2, 0)
