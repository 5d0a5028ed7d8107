"""The limit of a kernel's dynamic shared memory, against a stand-in for the runtime: no launch takes back what another has raised."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

SOURCE = r"""
#include <cassert>
#include <thread>
#include "smem_limit.h"
static int device = 0, sets = 0;
static bool refuse = false;
static std::map<std::pair<const void*, int>, int> now;
extern "C" cudaError_t CUDARTAPI cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t CUDARTAPI cudaGetLastError(void) { return cudaSuccess; }
extern "C" cudaError_t CUDARTAPI cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
  assert(a == cudaFuncAttributeMaxDynamicSharedMemorySize);
  if (refuse) return cudaErrorInvalidValue;
  ++sets;
  now[{f, device}] = v;
  return cudaSuccess;
}
int main() {
  const char k = 0, other = 0;
  assert(gb_allow_smem(&k, 16 * 1024) == 0 && sets == 0);                       // nothing to ask for
  assert((gb_allow_smem(&k, 48 * 1024) == 0 && now[{&k, 0}] == 48 * 1024));     // with static memory this is above the limit of a fresh kernel
  assert(gb_allow_smem(&k, 100000) == 0 && gb_allow_smem(&k, 200000) == 0 && gb_allow_smem(&k, 60000) == 0);
  assert((now[{&k, 0}] == 200000 && sets == 3));                                // raised twice more, never lowered
  assert((gb_allow_smem(&other, 60000) == 0 && now[{&other, 0}] == 60000));
  device = 1;                                                                   // a limit of its own
  assert((gb_allow_smem(&k, 60000) == 0 && now[{&k, 1}] == 60000 && now[{&k, 0}] == 200000));
  refuse = true;
  assert(gb_allow_smem(&k, 150000) == -10);
  refuse = false;
  assert((gb_allow_smem(&k, 150000) == 0 && now[{&k, 1}] == 150000));           // what was refused is asked for again
  device = 0;
  auto work = [&](size_t n) { for (int i = 0; i < 100000; ++i) { assert(gb_allow_smem(&other, n) == 0); } };
  std::thread a(work, 70000), b(work, 180000);
  a.join();
  b.join();
  assert((now[{&other, 0}] == 180000));
  return 0;
}
"""


@pytest.mark.skipif(not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime_api.h")) or not shutil.which("g++"), reason="needs g++ and CUDA's headers")
def test_limits_only_grow(tmp_path):
    (src := tmp_path / "t.cpp").write_text(SOURCE)
    inc = os.path.join(ROOT, "jdm-ghassan_v1_pro-_b200", "csrc", "cuda")
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I" + os.path.join(CUDA, "include"), "-I" + inc, str(src), "-o", exe], check=True)
    subprocess.run([exe], check=True, timeout=60)
