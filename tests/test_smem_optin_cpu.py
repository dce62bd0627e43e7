"""The dynamic shared memory opt-in is a setting of one device: the launchers'
helper sets it once on each, through a CUDA runtime of the test's own."""
import glob
import os
import re
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "pytorch-tcuscan_b200", "csrc")
CUDA = "/usr/local/cuda/include"

PROGRAM = r"""
#include "tcu_smem.h"
#include <cstdio>
#include <cstdlib>
static int dev = 0, calls = 0, fail = 0;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = dev; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute a, int v) {
  if (a != cudaFuncAttributeMaxDynamicSharedMemorySize || v != 65536) exit(2);
  ++calls;
  return fail ? cudaErrorInvalidValue : cudaSuccess;
}
static void kern_a(int) {}
static void kern_b(float) {}
static void want(int n, const char* what) { if (calls != n) { printf("%s: %d calls, not %d\n", what, calls, n); exit(1); } }
int main() {
  tcu::DeviceSet s, other;
  fail = 1;
  if (tcu::allow_smem(s, 65536, &kern_a, &kern_b) != cudaErrorInvalidValue) return 3;
  want(1, "a failure is reported at once");
  fail = 0;
  for (int pass = 0; pass < 3; ++pass)
    for (dev = 0; dev < 8; ++dev)
      if (tcu::allow_smem(s, 65536, &kern_a, &kern_b) != cudaSuccess) return 3;
  want(1 + 8 * 2, "both kernels once on each of 8 devices, also after the failure");
  dev = 3;
  tcu::allow_smem(other, 65536, &kern_a);
  want(1 + 8 * 2 + 1, "a launcher of its own");
  for (int pass = 0; pass < 2; ++pass)
    for (int d : {63, 64, 200}) { dev = d; tcu::allow_smem(other, 65536, &kern_a); }
  want(1 + 8 * 2 + 1 + 1 + 4, "device 63 once, those beyond the set every time");
  return 0;
}
"""


@pytest.mark.skipif(not shutil.which("g++") or not os.path.isdir(CUDA), reason="needs g++ and the CUDA headers")
def test_once_per_device(tmp_path):
    (tmp_path / "t.cpp").write_text(PROGRAM)
    r = subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-I", CUDA, str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_no_launcher_keeps_a_flag_per_process():
    for f in glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")):
        src = re.sub(r'"[^"\n]*"', "", open(f).read())
        assert not re.search(r"\bcudaFuncSetAttribute\s*\(", src), f
        assert not re.search(r"\bstatic\s+bool\s+\w+\s*=\s*false", src), f
