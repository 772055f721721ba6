"""Products around the number of tiles (8 of 128 x 64) from which they take the tcgen05 route, and far below one tile an
SM, against NumPy."""

import numpy as np
import pytest

from taurus_vap_gb300 import model as M
from taurus_vap_gb300.native import Context

pytestmark = pytest.mark.gpu


# 7, 8, 9 and 16 tiles of more than 1.2e7 multiply-adds; ragged rows, columns and lengths
@pytest.mark.parametrize("m,n,k", [(897 - 1, 64, 337), (1024, 61, 300), (1025, 64, 257), (513 - 1, 255, 161)])
@pytest.mark.parametrize("cplx", [False, True])
def test_few_tiles(m, n, k, cplx):
    ctx = Context(M.sd_model(seed=2).basis)
    rng = np.random.default_rng(m + n + k)

    def mat(r, c):
        x = rng.normal(size=(r, c))
        return x + 1j * rng.normal(size=(r, c)) if cplx else x

    A, B, C = mat(m, k), mat(k, n), mat(m, n)
    ref = A @ B
    big = lambda x, ax: np.maximum(np.abs(x.real), np.abs(x.imag)).max(axis=ax)  # noqa: E731
    # the documented bound of the emulated products, and the rounding of NumPy's own sum of K terms
    bound = (2.0 ** -46 if cplx else 2.0 ** -49) * k * np.outer(big(A, 1), big(B, 0)) + \
        4 * k * 2.0 ** -53 * (np.abs(A) @ np.abs(B))
    assert np.all(np.abs(ctx.gemm(A, B) - ref) <= bound)
    got = ctx.gemm(A, B, beta=0.5, C=C)
    assert np.all(np.abs(got - (ref + 0.5 * C)) <= bound + 2.0 ** -50 * (np.abs(ref) + np.abs(C)))
