"""csrc/smem_limit.h against a stand-in for the CUDA runtime: a kernel's limit is raised on every device that launches it, to the largest size asked for,
once; a call that fails is tried again; threads that ask for different sizes leave the larger one."""
import os
import subprocess

from qspec_b200 import build

PROGRAM = r"""
#include "smem_limit.h"
#include <stdio.h>
#include <thread>
#include <vector>
static thread_local int device = 0;
static std::atomic<int> calls{0}, fail{0}, limit[100];
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int bytes) {
  ++calls;
  if (fail) return cudaErrorInvalidValue;
  limit[device] = bytes;
  return cudaSuccess;
}
static void kernel() {}
#define CHECK(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
int main() {
  qspec::SmemLimit a;
  CHECK(a.raise(kernel, 60000) == cudaSuccess && limit[0] == 60000 && calls == 1);
  CHECK(a.raise(kernel, 60000) == cudaSuccess && a.raise(kernel, 50000) == cudaSuccess && calls == 1 && limit[0] == 60000);
  device = 1;
  CHECK(a.raise(kernel, 60000) == cudaSuccess && limit[1] == 60000 && calls == 2);
  device = 0;
  CHECK(a.raise(kernel, 90000) == cudaSuccess && limit[0] == 90000 && limit[1] == 60000 && calls == 3);
  device = 99;                                   // beyond what is remembered: asked every time
  CHECK(a.raise(kernel, 60000) == cudaSuccess && a.raise(kernel, 60000) == cudaSuccess && calls == 5 && limit[99] == 60000);
  device = 2;
  fail = 1;
  CHECK(a.raise(kernel, 60000) == cudaErrorInvalidValue);
  fail = 0;
  CHECK(a.raise(kernel, 60000) == cudaSuccess && limit[2] == 60000);
  for (int round = 0; round < 200; ++round) {
    qspec::SmemLimit b;
    std::vector<std::thread> threads;
    for (int i = 1; i <= 8; ++i) threads.emplace_back([&b, i] { device = 3; b.raise(kernel, 50000 + i); });
    for (auto& t : threads) t.join();
    CHECK(limit[3] == 50008);
    limit[3] = 0;
  }
  return 0;
}
"""


def test_limit_per_device(tmp_path):
    (tmp_path / "t.cpp").write_text(PROGRAM)
    cuda = os.path.dirname(os.path.dirname(build._nvcc())) or "/usr/local/cuda"
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{build.CSRC}", f"-I{cuda}/include", str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t"), "-lpthread"], check=True)
    run = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0, run.stdout


def test_no_launch_raises_a_limit_by_a_flag_of_its_own():
    """A static flag beside cudaFuncSetAttribute knows one device only."""
    for name in sorted(os.listdir(build.CSRC)):
        if name.endswith((".cu", ".cuh")):
            lines = open(os.path.join(build.CSRC, name)).read().splitlines()
            for i, line in enumerate(lines):
                if "cudaFuncSetAttribute" in line:
                    assert not any("static bool" in x or "static size_t" in x for x in lines[max(0, i - 3):i]), f"{name}:{i + 1}"
