"""The panels of the Gauss-Jordan solve (pivots in single precision, the block inverted in FP64) against the LU solve on
the FP64 pipe, for bases whose panels fill a warp's 32 rows, miss it by one quadruple, or pass it."""

import numpy as np
import pytest

from taurus_vap_gb300 import model as M
from taurus_vap_gb300.native import Context

pytestmark = pytest.mark.gpu

# n = 8, 28 and 32 (one panel), 36 (two of 18), 64 (two of 32), 68 (23, 23, 22), 96 (three of 32), 100 (four of 25)
SHELLS = {8: [103], 28: [307, 205], 32: [103, 205, 305], 36: [307, 205, 103], 64: [409, 307, 305, 205, 101],
          68: [409, 307, 305, 205, 103], 96: [409, 407, 307, 305, 205, 203, 103, 101],
          100: [409, 407, 307, 305, 205, 203, 103, 101, 1]}


@pytest.mark.parametrize("n", sorted(SHELLS))
def test_solve_panels(n):
    shells = SHELLS[n]
    mdl = M.synthetic(shells, [float(i) for i in range(len(shells))], hw=10.0, valence_Z=2, valence_N=2, seed=3,
                      damp=8.0)
    assert mdl.n == n
    U, V = M.random_bogoliubov(mdl.basis, 2, 2, seed=5)
    ctx = Context(mdl.basis, mdl.ham)
    res = []
    for mode in (0, 2):
        ctx.set_gemm_mode(mode)
        res.append(ctx.project(U, V, 5, 3, 2 * np.pi, 2, 2))
    (p0, h0), (p2, h2) = res
    e0, e2 = ((p.c("ener") / p.c("over")).real for p in (p0, p2))
    # the bounds of the comparison with the oracle at n = 24 .. 140
    assert abs(e0 - e2) < 1e-9 * max(1.0, abs(e0))
    assert abs(p0.c("over") - p2.c("over")) < 1e-10 * abs(p0.c("over")) + 1e-14
    assert np.linalg.norm(h2 - h0) < 1e-9 * np.linalg.norm(h0)


@pytest.mark.parametrize("grid", [17, 19])
def test_two_groups_of_angles(grid):
    # 145 and 181 folded angles: one group (at most one an SM), and two
    mdl = M.sd_model(seed=2)
    U, V = M.random_bogoliubov(mdl.basis, 4, 4, seed=3)
    ctx = Context(mdl.basis, mdl.ham)
    res = []
    for mode in (0, 2):
        ctx.set_gemm_mode(mode)
        res.append(ctx.project(U, V, grid, grid, 2 * np.pi, 4, 4))
    (p0, h0), (p2, h2) = res
    e0, e2 = ((p.c("ener") / p.c("over")).real for p in (p0, p2))
    assert abs(e0 - e2) < 1e-9 * max(1.0, abs(e0))
    assert np.linalg.norm(h2 - h0) < 1e-9 * np.linalg.norm(h0)
