"""The Thouless evolution against NumPy from the smallest basis over the largest of the Newton form (n = 224) to the
blocked form above it, for steps from tiny to so large that the FP32 start of the Newton form is of no use."""

import numpy as np
import pytest

from taurus_vap_gb300 import model as M
from taurus_vap_gb300.native import Context, TvapError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shells", [1, 2, 4, 5, 6, 9, 10, 15, 21, 22])
@pytest.mark.parametrize("scale", [0.0, 1e-4, 0.1, 3.0, 1e4])
def test_evolution(shells, scale):
    sh = M.shells_up_to(6)[:shells]
    n = 2 * sum(s % 100 + 1 for s in sh)
    mdl = M.synthetic(sh[:1], [1.0], hw=20.0, valence_Z=1, valence_N=1, seed=1)
    basis = mdl.basis
    for k in ("sp_n", "sp_l", "sp_2j", "sp_2mj", "sp_2mt", "sp_sh", "sp_tr"):
        setattr(basis, k, np.resize(getattr(basis, k), n))
    ctx = Context(basis)
    rng = np.random.default_rng(n)
    W = np.linalg.qr(rng.normal(size=(2 * n, n)))[0]
    U, V = W[:n], W[n:]
    B = rng.normal(size=(n, n))
    Z = scale * (B - B.T) / np.sqrt(2 * n)
    U1, V1 = ctx.evolve(U, V, Z)
    S = np.eye(n) + Z.T @ Z
    Li = np.linalg.inv(np.linalg.cholesky(S))
    # normwise forward error of an n x n triangular inverse and the products with it, on both sides
    tol = 16 * n * 2.0 ** -53 * np.linalg.cond(S)
    for got, A in ((U1, U + V @ Z), (V1, V + U @ Z)):
        assert np.linalg.norm(got - A @ Li.T) <= tol * np.linalg.norm(A @ Li.T) + 1e-300


def test_non_finite_step_is_reported():
    mdl = M.sd_model(seed=2)
    ctx = Context(mdl.basis)
    U, V = M.random_bogoliubov(mdl.basis, 4, 4, seed=3)
    Z = np.zeros((mdl.n, mdl.n))
    Z[0, 1] = np.nan
    with pytest.raises(TvapError) as e:
        ctx.evolve(U, V, Z)
    assert e.value.code == 14
    assert np.all(np.isfinite(ctx.evolve(U, V, 0 * np.eye(mdl.n))[0]))
