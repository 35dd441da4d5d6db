"""Phase timing where the host runs out of memory: a phase that finds no memory for its record is left
out, the call goes on, and no exception leaves a kernel running that stores to the call's memory.  A
program whose operator new fails on request makes every allocation of a call fail in turn."""
import os
import shutil
import subprocess

import pytest

import atc
import oracle
from conftest import ROOT

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <new>
#include <vector>
#include "atc.h"

static thread_local int left = -1;  // allocations until one fails; -1: none does
void* operator new(std::size_t n) {
  if (left > 0 && --left == 0) { left = -1; throw std::bad_alloc(); }
  if (void* p = std::malloc(n ? n : 1)) return p;
  throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }

static bool fails_with(int n, atc_status got, atc_status a, atc_status b) {
  if (got == a || got == b) return false;
  std::printf("allocation %d: status %d: %s\n", n, (int)got, atc_last_error());
  return true;
}

int main(int argc, char** argv) {
  if (argc < 2 || atc_init(0) != ATC_OK) return 2;
  uint64_t pairs = 0, want = 0, got = 0;
  if (atc_read_edges(argv[1], nullptr, 0, &pairs) != ATC_OK) return 2;
  std::vector<int32_t> e(2 * pairs);
  if (atc_read_edges(argv[1], e.data(), pairs, &pairs) != ATC_OK) return 2;
  // a call with no device work: its only allocation is the phase's record
  atc_csr none{};
  atc_phase_timing(1);
  left = 1;
  atc_status st = atc_kcl(&none, 4, &got, nullptr, nullptr);
  left = -1;
  if (fails_with(1, st, ATC_OK, ATC_OK)) return 1;
  atc_phase_timing(0);
  atc_csr csr{};
  if (atc_pretc(e.data(), pairs, ATC_DIR_DEGREE, ATC_ORDER_NONE, nullptr, &csr, nullptr, nullptr) != ATC_OK) return 2;
  if (atc_tc(&csr, ATC_KERNEL_HU, nullptr, &want, nullptr, nullptr) != ATC_OK) return 2;
  for (int n = 1; n <= 12; ++n) {
    atc_phase_timing(1);
    left = n;
    st = atc_tc(&csr, ATC_KERNEL_HU, nullptr, &got, nullptr, nullptr);
    left = -1;
    atc_phase_timing(0);
    if (fails_with(n, st, ATC_OK, ATC_ERR_OOM)) return 1;
    if (st == ATC_OK && got != want) return 1;
    if (atc_tc(&csr, ATC_KERNEL_HU, nullptr, &got, nullptr, nullptr) != ATC_OK || got != want) return 1;
  }
  atc_csr_free(&csr);
  std::printf("count %llu\n", (unsigned long long)want);
  return 0;
}
"""


def test_phase_without_memory(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    (tmp_path / "p.cpp").write_text(PROGRAM)
    g = atc.rmat_graph(9, 8, 4)
    g.tofile(tmp_path / "g.bin")
    libdir = os.path.dirname(atc.LIB_PATH)
    exe = tmp_path / "p"
    r = subprocess.run([cxx, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "include"), str(tmp_path / "p.cpp"), "-o",
                        str(exe), "-L", libdir, "-latc", "-Wl,-rpath," + libdir], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe), str(tmp_path / "g.bin")], capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)
    assert "count %d" % oracle.tc_count(g) in r.stdout
