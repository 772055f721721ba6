"""The Thouless evolution where its cooperative launch does not run: the single-CTA inverse works on the products of this
call, for every basis size, also those whose products the launch would have formed itself."""

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, os.pardir, "taurus_vap_gb300", "csrc")


def test_products_are_formed_before_they_are_read(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", CSRC, "-I", os.path.join(HERE, os.pardir, "include"),
                    os.path.join(HERE, "evolve_route_check.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and "bad 0" in out.stdout, out.stdout + out.stderr
    # the evolution takes that route
    assert "evolve_route(evolve_forms_products(n), products, coop, single)" in \
        open(os.path.join(CSRC, "gradient.cu")).read()
