"""The fields of a few density columns (gather_few_kernel) against the oracle: the column counts around every split of
a warp into columns and slots, and the first counts of the paths on either side."""

import numpy as np
import pytest

import oracle as O
from taurus_vap_gb300 import model as M
from taurus_vap_gb300.native import Context

pytestmark = pytest.mark.gpu

FIELD_TOL = 1e-12  # relative to the largest entry (the accuracy the fields must keep)


@pytest.mark.parametrize("mode", [0, 2])
@pytest.mark.parametrize("space", ["sd", "emax2"])
def test_few_columns(space, mode):
    mdl = M.sd_model(seed=2) if space == "sd" else M.noncore_model(2, seed=5, valence_Z=4, valence_N=4)
    om, ctx, n = O.OracleModel(mdl), Context(mdl.basis, mdl.ham), mdl.n
    ctx.set_gemm_mode(mode)
    rng = np.random.default_rng(11)
    c = lambda: rng.normal(size=(17, n, n)) + 1j * rng.normal(size=(17, n, n))  # noqa: E731
    rho, kl, kr = c(), c(), c()
    kl, kr = kl - kl.transpose(0, 2, 1), kr - kr.transpose(0, 2, 1)
    ref = [om.calculate_fields(rho[q], kl[q], kr[q], nthreads=1) for q in range(17)]
    for cols in (1, 2, 3, 4, 5, 8, 9, 15, 16, 17):
        got = ctx.calculate_fields_batched(rho[:cols], kl[:cols], kr[:cols])
        for k in range(4):
            for q in range(cols):
                assert np.abs(got[k][q] - ref[q][k]).max() <= FIELD_TOL * np.abs(ref[q][k]).max(), (cols, k, q)
