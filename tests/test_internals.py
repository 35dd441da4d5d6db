"""Sections of tests/internals/internals.cu, which includes the library's sources: parts that no call
reaches at a test's size, and rules that show in times only."""
import os
import shutil
import subprocess

import pytest

import atc
from conftest import ROOT

CSRC = os.path.join(ROOT, "accelerating-tc_gb300", "csrc")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    exe = tmp_path_factory.mktemp("internals") / "internals"
    libdir = os.path.dirname(atc.LIB_PATH)
    r = subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O1", "-std=c++17",
                        "--expt-relaxed-constexpr", "-I", os.path.join(ROOT, "include"), "-I", CSRC,
                        os.path.join(ROOT, "tests", "internals", "internals.cu"), "-o", str(exe), "-L", libdir, "-latc",
                        "-Xlinker", "-rpath", "-Xlinker", libdir], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return exe


def _run(program, section):
    r = subprocess.run([str(program), section], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout == "ok\n", (r.returncode, r.stdout, r.stderr)


def test_batch_shapes(program):
    _run(program, "shapes")
