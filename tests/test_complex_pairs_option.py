"""TVAP_OPT_COMPLEX_PAIRS: 0 switches the paired form off, k > 0 takes it from contraction length k on, and a new context
has 81.  (The bits do not show the form, so the rule itself is checked, on the host.)"""

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, os.pardir, "taurus_vap_gb300", "csrc")
CUDA_INCLUDE = "/usr/local/cuda/include"


def test_rule(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None or not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h")):
        pytest.skip("no C++ compiler or no CUDA headers")
    exe = tmp_path / "check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", CSRC, "-I", os.path.join(HERE, os.pardir, "include"), "-I",
                    CUDA_INCLUDE, os.path.join(HERE, "pairs_rule_check.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and "bad 0" in out.stdout, out.stdout + out.stderr
    # and the product asks that rule, with what the context holds
    src = open(os.path.join(CSRC, "ozaki.cu")).read()
    assert "&& complex_pairs(K, g_tc_pairs_min_k);" in src


@pytest.mark.gpu
def test_option_of_a_context():
    from taurus_vap_gb300 import model as M
    from taurus_vap_gb300.native import Context

    ctx = Context(M.sd_model(seed=2).basis)
    default = ctx.option(ctx.OPT_COMPLEX_PAIRS)
    assert default == 81
    ctx.set_option(ctx.OPT_COMPLEX_PAIRS, 0)
    assert ctx.option(ctx.OPT_COMPLEX_PAIRS) == 0
    ctx.set_option(ctx.OPT_COMPLEX_PAIRS, default)
    assert ctx.option(ctx.OPT_COMPLEX_PAIRS) == default
