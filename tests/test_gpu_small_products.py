"""Products up to the size that runs on the FP64 pipe in every mode (small_gemm_kernel), against NumPy: edges of the
8 x 8 tiles and of the staged k range, every transposition, conjugation, alpha and beta."""

import numpy as np
import pytest

from taurus_vap_gb300 import model as M
from taurus_vap_gb300.native import Context

pytestmark = pytest.mark.gpu

SIZES = [(1, 1, 1), (7, 9, 2), (8, 8, 95), (9, 7, 96), (17, 16, 97), (24, 24, 128), (33, 5, 129), (40, 41, 257),
         (140, 140, 140), (3, 200, 1000), (100000, 1, 3)]


@pytest.fixture(scope="module")
def ctx():
    return Context(M.sd_model(seed=2).basis)


@pytest.mark.parametrize("m,n,k", SIZES)
@pytest.mark.parametrize("cplx", [False, True])
def test_small_products(ctx, m, n, k, cplx):
    rng = np.random.default_rng(m + 3 * n + 7 * k)

    def mat(r, c):
        x = rng.normal(size=(r, c)) * 10.0 ** rng.integers(-3, 4, size=(r, 1))
        return x + 1j * rng.normal(size=(r, c)) if cplx else x

    op = {"N": lambda x: x, "T": lambda x: x.T, "C": lambda x: x.conj().T}
    for ta, tb in [("N", "N"), ("T", "N"), ("N", "T"), ("C", "T"), ("T", "C")]:
        A = mat(m, k) if ta == "N" else mat(k, m)
        B = mat(k, n) if tb == "N" else mat(n, k)
        C = mat(m, n)
        alpha, beta = (0.5 - 0.25j, 2.0 + 1.0j) if cplx else (-1.5, 0.5)
        a, b = op[ta](A), op[tb](B)
        got = ctx.gemm(A, B, ta, tb, alpha, beta, C)
        ref = alpha * (a @ b) + beta * C
        # any order of the K multiply-adds and the two scalings: (K + 4) roundings of terms that sum to |A||B| and
        # |C|, a complex term being four real products; on both sides
        u = 2.0 ** -53 * (k + 4) * (4 if cplx else 1) * 2
        bound = u * (abs(alpha) * (np.abs(a) @ np.abs(b)) + abs(beta) * np.abs(C))
        assert np.all(np.abs(got - ref) <= bound), (ta, tb, float((np.abs(got - ref) / bound).max()))
