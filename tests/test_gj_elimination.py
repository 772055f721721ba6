"""The elimination product of the Thouless solve writes into the matrix that holds its operands: on the host, that it
reads nothing it writes (taurus_vap_gb300/csrc/gj_elimination.h), and that every kernel on the FP64 pipe asks."""

import os
import re
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, os.pardir, "taurus_vap_gb300", "csrc")
CUDA_INCLUDE = "/usr/local/cuda/include"


def test_reads_and_writes_are_disjoint(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None or not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h")):
        pytest.skip("no C++ compiler or no CUDA headers")
    exe = tmp_path / "check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", CSRC, "-I", os.path.join(HERE, os.pardir, "include"), "-I",
                    CUDA_INCLUDE, os.path.join(HERE, "gj_elimination_check.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and "bad 0" in out.stdout, out.stdout + out.stderr


def test_every_fp64_kernel_leaves_the_kept_rows():
    src = open(os.path.join(CSRC, "dense.cu")).read()
    bodies = re.split(r"__global__", src)
    kernels = [b for b in bodies[1:] if re.match(r"[^;{]*\bGemmArgs g\b", b)]
    assert len(kernels) == 3
    assert all("g.writes_row(" in b for b in kernels)
