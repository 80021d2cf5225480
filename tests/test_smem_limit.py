"""A kernel's shared memory limit is raised once on every device of a process
(harm_smem.h, compiled against a stand-in for the CUDA runtime): a limit
raised for the first device only leaves launches on a second one refused."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "harm_ramt_b200", "csrc")

RUNTIME = """
#pragma once
enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidValue = 1 };
enum cudaFuncAttribute { cudaFuncAttributeMaxDynamicSharedMemorySize = 8 };
extern int device, calls, refuse, limit[128];
inline cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
inline cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int bytes)
{
  calls++;
  if (refuse) return cudaErrorInvalidValue;
  limit[device] = bytes;
  return cudaSuccess;
}
"""
MAIN = """
#include <cstdio>
#include "harm_smem.h"
int device = 0, calls = 0, refuse = 0, limit[128];
int main()
{
  static harm::SmemLimit s, other;
  const int devices[] = {0, 1, 0, 3, 63, 64, 1, 64};
  for (int d : devices) {
    device = d;
    s.raise(&s, 99000);
    if (limit[d] != 99000) return 1;
  }
  if (calls != 6) return 2;  // 0, 1, 3, 63 once each, 64 at every launch
  device = 5;
  refuse = 1;
  s.raise(&s, 99000);
  refuse = 0;
  s.raise(&s, 99000);
  if (limit[5] != 99000) return 3;
  device = 0;
  other.raise(&other, 50000);
  return (limit[0] == 50000) ? 0 : 4;
}
"""


def test_raised_on_every_device(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text(RUNTIME)
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = str(tmp_path / "a.out")
    subprocess.run(["g++", "-std=c++17", "-I", str(tmp_path), "-I", CSRC, "-o", exe, str(tmp_path / "main.cpp")], check=True)
    assert subprocess.run([exe]).returncode == 0


def test_every_raised_limit_goes_through_it():
    """No launcher of the step raises a limit behind a flag of the process."""
    for f in os.listdir(CSRC):
        if f != "harm_smem.h" and f.endswith((".cu", ".cuh", ".h")):
            assert "cudaFuncSetAttribute" not in open(os.path.join(CSRC, f)).read(), f
