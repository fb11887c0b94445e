"""Kernels that want more than 48 KB of shared memory are allowed it on every device of a process."""
import subprocess

PROGRAM = r"""
#include "device_attr.h"
#include <initializer_list>
static int device = 0, calls[80], carveouts[80], failing = 0;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute a, int) {
  if (failing) return cudaErrorInvalidValue;
  ++(a == cudaFuncAttributeMaxDynamicSharedMemorySize ? calls : carveouts)[device];
  return cudaSuccess;
}
static void kernel() {}
static int launch(int d, int bytes = 100 * 1024) {
  static CbDeviceAttr attr;
  device = d;
  return cb_allow_smem(attr, kernel, bytes, true);
}
int main() {
  failing = 1;
  int wrong = launch(0) == 0;                                        // a refusal is handed on, and asked again
  failing = 0;
  for (int turn = 0; turn < 3; ++turn)
    for (int d : {0, 1, 7, 63}) wrong |= launch(d) != 0;
  for (int d : {0, 1, 7, 63}) wrong |= calls[d] != 1 || carveouts[d] != 1;
  for (int turn = 0; turn < 2; ++turn) wrong |= launch(70) != 0;
  wrong |= calls[70] != 2;
  static CbDeviceAttr small;
  device = 2;
  wrong |= cb_allow_smem(small, kernel, 48 * 1024) != 0 || calls[2] != 0 || carveouts[2] != 0;
  return wrong;
}
"""


def test_said_once_on_each_device(tmp_path):
    from colossalai_b200.kernel.loader import CSRC

    src, exe = tmp_path / "attr.cpp", tmp_path / "attr"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", str(CSRC), "-I", "/usr/local/cuda/include", str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0


def test_no_kernel_says_it_by_itself():
    from colossalai_b200.kernel.loader import CSRC

    for f in [*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]:
        assert "cudaFuncSetAttribute" not in f.read_text(), f.name
