"""kernel_limits (csrc/sgh_limits.h) against a fake of the runtime's two calls, on
the CPU: a kernel's limit is raised on every device that uses it, is never
lowered, and covers each caller's own size while other threads ask for
others; an error is returned and not remembered."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "spectral_galerkin_heat_b200", "csrc")
CUDA = "/usr/local/cuda/include"

PROGRAM = r"""
#include <atomic>
#include <cstdio>
#include <map>
#include <thread>
#include <vector>
#include "sgh_limits.h"

static thread_local int device = 0;
static std::mutex m;
static std::map<std::pair<const void*, int>, int> bytes_of, wide_of;
static std::atomic<int> calls{0};
static bool refuse = false;

extern "C" cudaError_t CUDARTAPI cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t CUDARTAPI cudaFuncSetAttribute(const void* f, enum cudaFuncAttribute a, int v) {
  ++calls;
  if (refuse) return cudaErrorInvalidValue;
  std::lock_guard<std::mutex> g(m);
  (a == cudaFuncAttributeNonPortableClusterSizeAllowed ? wide_of : bytes_of)[{f, device}] = v;
  return cudaSuccess;
}
static int limit(const void* f) { std::lock_guard<std::mutex> g(m); return bytes_of[{f, device}]; }
#define CHECK(x) do { if (!(x)) { std::printf("failed: %s\n", #x); return 1; } } while (0)

int main() {
  const char k[3] = {};
  CHECK(sgh::kernel_limits(&k[0], 90000) == cudaSuccess && limit(&k[0]) == 90000);
  CHECK(sgh::kernel_limits(&k[0], 60000) == cudaSuccess && limit(&k[0]) == 90000);   // never lowered
  CHECK(calls == 1);
  CHECK(sgh::kernel_limits(&k[0], 100000, true) == cudaSuccess && limit(&k[0]) == 100000 && calls == 3);
  device = 1;  // a second device of the process starts from its own default
  CHECK(limit(&k[0]) == 0);
  CHECK(sgh::kernel_limits(&k[0], 60000, true) == cudaSuccess && limit(&k[0]) == 60000);
  CHECK((wide_of[{&k[0], 1}] == 1));
  device = 0;
  refuse = true;
  CHECK(sgh::kernel_limits(&k[1], 80000) == cudaErrorInvalidValue);
  refuse = false;
  CHECK(sgh::kernel_limits(&k[1], 80000) == cudaSuccess && limit(&k[1]) == 80000);
  std::atomic<int> bad{0};
  std::vector<std::thread> ts;
  for (int t = 0; t < 4; ++t)
    ts.emplace_back([&, t] {
      for (int i = 0; i < 20000; ++i) {
        const int b = 50000 + 100 * ((i * 7 + t * 13) % 400);
        if (sgh::kernel_limits(&k[2], b) != cudaSuccess || limit(&k[2]) < b) ++bad;
      }
    });
  for (auto& t : ts) t.join();
  CHECK(bad == 0);
  std::puts("ok");
  return 0;
}
"""


@pytest.mark.skipif(not os.path.exists(os.path.join(CUDA, "cuda_runtime_api.h")) or shutil.which("g++") is None,
                    reason="needs the CUDA headers and g++")
def test_limits_only_grow_per_kernel_and_device(tmp_path):
    src, exe = tmp_path / "limits.cpp", tmp_path / "limits"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, "-I", CUDA, str(src), "-o", str(exe)],
                   check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout


def test_no_kernel_sets_its_limits_any_other_way():
    """A limit raised once per process would hold on the first device only."""
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh", ".h")) and name != "sgh_limits.h":
            text = open(os.path.join(CSRC, name)).read()
            assert "cudaFuncSetAttribute" not in text, name
