"""Which products run on the FP64 pipe (taurus_vap_gb300/csrc/gemm_route.h): on the host, the rule against measured
times of both sides; on the device, products on either side of its lines against NumPy."""

import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, os.pardir, "taurus_vap_gb300", "csrc")


def test_rule_takes_the_faster_side(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", CSRC, os.path.join(HERE, "gemm_route_check.cpp"), "-o", str(exe)],
                   check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and "bad 0" in out.stdout, out.stdout + out.stderr


# short lengths (FP64 tiles beyond few outputs), lengths from 16 on with few and many tiles, small and larger batches of
# the real representation's tiles (7 and 8 of 128 x 64), a length that the slicing pass cannot hold
@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(300, 200, 3), (1100, 1100, 3), (400, 400, 8), (450, 450, 15), (450, 450, 16),
                                   (512, 256, 28), (300, 300, 28), (250, 190, 70), (448, 128, 40), (513, 128, 40),
                                   (40, 40, 2000)])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("gemm_mode", [0, 1, 2])
def test_both_sides(m, n, k, cplx, gemm_mode):
    from taurus_vap_gb300 import model as M
    from taurus_vap_gb300.native import Context

    ctx = Context(M.sd_model(seed=2).basis)
    ctx.set_gemm_mode(gemm_mode)
    rng = np.random.default_rng(m + n + k)

    def mat(r, c):
        x = rng.normal(size=(r, c))
        return x + 1j * rng.normal(size=(r, c)) if cplx else x

    A, B, C = mat(m, k), mat(k, n), mat(m, n)
    ref = A @ B
    big = lambda x, ax: np.maximum(np.abs(x.real), np.abs(x.imag)).max(axis=ax)  # noqa: E731
    # the documented bound of the emulated products, and two sums of K terms in any order (complex: four real ones)
    bound = (2.0 ** -46 if cplx else 2.0 ** -49) * k * np.outer(big(A, 1), big(B, 0)) + \
        2 * (k + 4) * (4 if cplx else 1) * 2.0 ** -53 * (np.abs(A) @ np.abs(B))
    assert np.all(np.abs(ctx.gemm(A, B) - ref) <= bound)
    got = ctx.gemm(A, B, beta=-2.0, C=C)
    assert np.all(np.abs(got - (ref - 2.0 * C)) <= bound + 2.0 ** -50 * (np.abs(ref) + 2 * np.abs(C)))
