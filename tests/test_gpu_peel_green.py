"""The peels on a stream with few SMs (a green context's): their blocks must all be resident, so fewer of
them are launched, and the results are those of the whole device."""
import os
import shutil
import subprocess

import pytest

import atc
from conftest import ROOT

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <cuda.h>
#include <cstdio>
#include <cstring>
#include <vector>
#include "atc.h"

#define DRV(call)                                                          \
  do {                                                                     \
    CUresult r_ = (call);                                                  \
    if (r_ != CUDA_SUCCESS) {                                              \
      std::printf("unavailable: %s: %d\n", #call, (int)r_);                \
      return 3;                                                            \
    }                                                                      \
  } while (0)
#define LIB(call)                                                          \
  do {                                                                     \
    if ((call) != ATC_OK) {                                                \
      std::printf("%s: %s\n", #call, atc_last_error());                    \
      return 1;                                                            \
    }                                                                      \
  } while (0)

int main() {
  LIB(atc_init(0));
  CUdevice dev;
  DRV(cuInit(0));
  DRV(cuDeviceGet(&dev, 0));
  CUdevResource all, part;
  DRV(cuDeviceGetDevResource(dev, &all, CU_DEV_RESOURCE_TYPE_SM));
  unsigned groups = 1;
  DRV(cuDevSmResourceSplitByCount(&part, &groups, &all, nullptr, 0, 16));
  CUdevResourceDesc desc;
  DRV(cuDevResourceGenerateDesc(&desc, &part, 1));
  CUgreenCtx ctx;
  DRV(cuGreenCtxCreate(&ctx, desc, dev, CU_GREEN_CTX_DEFAULT_STREAM));
  CUstream s;
  DRV(cuGreenCtxStreamCreate(&s, ctx, CU_STREAM_NON_BLOCKING, 0));
  const uint32_t scale = 15, ef = 16;
  const uint64_t pairs = (uint64_t)ef << scale;
  std::vector<int32_t> e(2 * pairs);
  LIB(atc_gen_rmat_host(scale, ef, 570000, 190000, 190000, 3, e.data(), 4));
  std::vector<int32_t> out[2], prio[2];
  std::vector<uint64_t> packed(pairs), cores[2];
  std::vector<int32_t> core[2];
  for (uint64_t i = 0; i < pairs; ++i) packed[i] = (uint64_t)(uint32_t)e[2 * i] << 32 | (uint32_t)e[2 * i + 1];
  for (int q = 0; q < 2; ++q) {
    uint64_t n = 0, nv = 0;
    out[q].assign(4 * pairs, 0);
    prio[q].assign(1u << scale, 0);
    cores[q].assign(pairs, 0);
    core[q].assign(1u << scale, 0);
    LIB(atc_adirection(e.data(), pairs, out[q].data(), &n, prio[q].data(), q ? (atc_stream)s : nullptr));
    LIB(atc_kcore_direction(packed.data(), pairs, cores[q].data(), core[q].data(), &nv, q ? (atc_stream)s : nullptr));
  }
  if (out[0] != out[1] || prio[0] != prio[1] || cores[0] != cores[1] || core[0] != core[1]) {
    std::printf("results differ\n");
    return 1;
  }
  DRV(cuStreamDestroy(s));
  DRV(cuGreenCtxDestroy(ctx));
  std::printf("equal on %u of %u SMs\n", part.sm.smCount, all.sm.smCount);
  return 0;
}
"""


def test_peels_on_few_sms(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    cuda = "/usr/local/cuda"
    if cxx is None or not os.path.exists(cuda + "/include/cuda.h"):
        pytest.skip("no C++ compiler or no cuda.h")
    (tmp_path / "p.cpp").write_text(PROGRAM)
    libdir = os.path.dirname(atc.LIB_PATH)
    exe = tmp_path / "p"
    stubs = next((d for d in (cuda + "/lib64/stubs", cuda + "/targets/sbsa-linux/lib/stubs") if os.path.isdir(d)), ".")
    r = subprocess.run([cxx, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "include"), "-I", cuda + "/include",
                        str(tmp_path / "p.cpp"), "-o", str(exe), "-L", libdir, "-latc", "-Wl,-rpath," + libdir,
                        "-L", stubs, "-lcuda"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    if r.returncode == 3:
        pytest.skip(r.stdout)
    assert r.returncode == 0 and "equal on" in r.stdout, (r.returncode, r.stdout, r.stderr)
