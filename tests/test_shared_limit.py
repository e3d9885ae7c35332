"""The limit of dynamic shared memory, raised once per kernel and device: the header against a fake of the runtime, on the CPU."""
import os
import subprocess

from torch.utils.cpp_extension import CUDA_HOME

PROGRAM = r"""
#include "shared_limit.h"
#include <cstdio>
static int device = 0, calls[80], bytes_seen = 0;
static bool fails = false;
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute a, int v) {
  if (a != cudaFuncAttributeMaxDynamicSharedMemorySize) return cudaErrorInvalidValue;
  ++calls[device];
  bytes_seen = v;
  return fails ? cudaErrorInvalidValue : cudaSuccess;
}
int main() {
  tb::SharedLimit a, b;
  int kernel = 0;
  auto raise = [&](tb::SharedLimit& l, int d) { device = d; return l.raise(&kernel, 1000) == cudaSuccess; };
  bool ok = raise(a, 0) && raise(a, 0) && raise(a, 0) && calls[0] == 1 && bytes_seen == 1000;   // once on a device
  ok = ok && raise(a, 3) && raise(a, 3) && calls[3] == 1 && raise(a, 0) && calls[0] == 1;       // and once on the next
  ok = ok && raise(a, 63) && raise(a, 63) && calls[63] == 1;
  ok = ok && raise(b, 0) && calls[0] == 2;                                                       // another kernel
  fails = true;
  ok = ok && !raise(a, 5) && !raise(a, 5) && calls[5] == 2;                                      // a failure is not remembered
  fails = false;
  ok = ok && raise(a, 5) && raise(a, 5) && calls[5] == 3;
  ok = ok && raise(a, 70) && raise(a, 70) && calls[70] == 2 && raise(a, 6) && calls[6] == 1;     // more devices than bits
  std::puts(ok ? "ok" : "wrong");
}
"""


def test_once_per_device(tmp_path):
    from terra_b200 import _ext

    src, exe = tmp_path / "limit.cpp", tmp_path / "limit"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", _ext.CSRC, "-I", os.path.join(CUDA_HOME, "include"), "-o", exe, src], check=True)
    assert subprocess.run([exe], capture_output=True, text=True, check=True).stdout.strip() == "ok"


def test_every_limit_of_a_common_launch_goes_through_it():
    from terra_b200 import _ext

    for name in ("elementwise.cu", "gemm_sm100.cu", "window_attn.cu"):
        with open(os.path.join(_ext.CSRC, name)) as f:
            assert "cudaFuncSetAttribute" not in f.read(), name
