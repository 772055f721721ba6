"""The <O^2> sums for operators at and beyond the limit of the sparse form (8 entries a row or column), against the
oracle with the bounds of the other observables."""

import math

import numpy as np
import pytest

from taurus_vap_gb300 import model as M
from taurus_vap_gb300.native import Context

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("entries", [8, 9, 12])
def test_squares_by_entries_per_row(entries):
    mdl = M.sd_model(seed=2)
    U, V = M.random_bogoliubov(mdl.basis, 4, 4, seed=3)
    ops = dict(mdl.observable_operators())
    n, h = mdl.n, mdl.n // 2
    rng = np.random.default_rng(entries)
    i, j = np.indices((n, n))
    away = np.minimum((i - j) % h, (j - i) % h)
    # real symmetric, within an isospin, `entries` in every row and column
    band = (i // h == j // h) & {8: (away >= 1) & (away <= 4), 9: away <= 4, 12: away >= 0}[entries]
    assert np.all(band.sum(0) == entries) and np.all(band.sum(1) == entries)

    def operator():
        B = rng.normal(size=(n, n))
        return np.where(band, B + B.T, 0.0).astype(np.complex128)

    ops["sq"] = np.array([(operator(), operator()), tuple(ops["sq"][0])])
    args = (U, V, 5, 5, 2 * math.pi, 4, 4, ops)
    ref = O.OracleModel(mdl).project_observables(*args, with_parity=False)
    got = Context(mdl.basis, mdl.ham).project_observables(*args, with_parity=False)
    assert ref["status"] == 0
    x, y = np.asarray(got["sq"]) / got["scal"][0], np.asarray(ref["sq"]) / ref["scal"][0]
    assert np.all(np.abs(x - y) <= 1e-9 * (1.0 + np.abs(y)))
