"""The opt-in to large dynamic shared memory is per kernel and device: a process
that launches on a second device has to set it there too.  The helper is compiled
here with a fake of the two runtime calls; no GPU is needed."""

import re
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "learning-based-attention-kernel-regression_b200" / "csrc"

PROGRAM = r"""
#include "smem_optin.cuh"
#include <cstdio>
#include <thread>
#include <vector>
static thread_local int device = 0;
static std::atomic<int> calls[66];
static std::atomic<int> failures{0};
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void*, enum cudaFuncAttribute, int bytes) {
  if (bytes != 200 * 1024) return cudaErrorInvalidValue;
  if (failures > 0) { --failures; return cudaErrorInvalidValue; }
  ++calls[device];
  return cudaSuccess;
}
static void kernel_a() {}
static void kernel_b() {}
#define CHECK(x) if (!(x)) { std::printf("failed: %s\n", #x); return 1; }
int main() {
  laker::SmemOptIn a, b;
  failures = 1;
  CHECK(a.allow(kernel_a, 200 * 1024) == cudaErrorInvalidValue);  // not remembered
  for (int i = 0; i < 3; ++i) CHECK(a.allow(kernel_a, 200 * 1024) == cudaSuccess);
  CHECK(calls[0] == 1);
  device = 1;
  for (int i = 0; i < 3; ++i) CHECK(a.allow(kernel_a, 200 * 1024) == cudaSuccess);
  CHECK(calls[1] == 1);
  CHECK(b.allow(kernel_b, 200 * 1024) == cudaSuccess);  // its own kernel
  CHECK(calls[1] == 2);
  device = 65;  // past the remembered ones: set at each call
  for (int i = 0; i < 3; ++i) CHECK(a.allow(kernel_a, 200 * 1024) == cudaSuccess);
  CHECK(calls[65] == 3);
  std::vector<std::thread> ts;
  for (int t = 0; t < 8; ++t)
    ts.emplace_back([&, t] {
      device = 8 + t;
      for (int i = 0; i < 1000; ++i) a.allow(kernel_a, 200 * 1024);
    });
  for (auto& t : ts) t.join();
  for (int t = 0; t < 8; ++t) CHECK(calls[8 + t] == 1);
  return 0;
}
"""


def test_opt_in_is_set_once_on_each_device(tmp_path):
    cuda = Path("/usr/local/cuda/include")
    if not shutil.which("g++") or not (cuda / "cuda_runtime_api.h").exists():
        pytest.skip("no host compiler or CUDA headers")
    (tmp_path / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-pthread", f"-I{CSRC}", f"-I{cuda}", "-o",
                    str(tmp_path / "t"), str(tmp_path / "t.cpp")], check=True)
    out = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout


def test_no_launcher_remembers_the_opt_in_for_the_process():
    for src in CSRC.glob("*.cu"):
        text = src.read_text()
        # a flag of the process in front of the call
        assert not re.search(r"static\s+bool\s+\w+[^;]*;[^}]*cudaFuncSetAttribute", text), src.name
