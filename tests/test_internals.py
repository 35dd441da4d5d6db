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


def test_batch_choice(program):
    """Also the benchmark's copy of the rule, on the same batches."""
    _run(program, "choice")
    import bench
    for graphs, n, m, w, wmin, longest, rows in ((1, 1048576, 15701789, 286.8, 127.6, 615, False),
                                                 (1, 1048576, 4087819, 94.7, 39.3, 200, True),
                                                 (6, 1048576, 4087656, 96.1, 39.7, 204, False),
                                                 (48, 20000, 357849, 29.1, 18.9, 54, True)):
        assert bench.rows_graphs([(m, w * m, wmin * m, n, longest)] * graphs) == [rows] * graphs
    assert bench.rows_graphs([]) == []


def test_barrier_wait_counts_polls(program):
    _run(program, "wait")


@pytest.mark.gpu
@pytest.mark.parametrize("section", ["sorts", "rows", "peel"])
def test_on_the_device(program, section):
    _run(program, section)
