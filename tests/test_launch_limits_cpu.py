"""CPU: how the launch sites raise a kernel's shared-memory limit, against a stand-in for the CUDA runtime."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "causal-flare_b200", "csrc")

SOURCE = r"""
#include "flare_common.cuh"
static int limit = 48 * 1024, asked = 0;
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int value) {
  limit = value;
  ++asked;
  return cudaSuccess;
}
static void kernel_of_two_launch_sites() {}
extern "C" int limit_after_a_launch() {
  if (flare::allow_smem(kernel_of_two_launch_sites) != cudaSuccess) return -1;
  return limit;
}
extern "C" void rebuild_context() { limit = 48 * 1024; }
extern "C" int times_asked() { return asked; }
"""

# what nvcc's start-up code calls in the runtime that is not linked here
STUBS = """
void** __cudaRegisterFatBinary(void* f) { return (void**)f; }
void __cudaRegisterFatBinaryEnd(void** h) {}
void __cudaUnregisterFatBinary(void** h) {}
char __cudaInitModule(void** h) { return 0; }
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    d = tmp_path_factory.mktemp("fake_runtime")
    (d / "t.cu").write_text(SOURCE)
    (d / "stubs.c").write_text(STUBS)
    cmd = [nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-Xcompiler", "-fPIC", "-shared", "-cudart", "none",
           "-Xlinker", "-Bsymbolic",  # (a CUDA runtime that the test process has loaded must not take the stand-in's place)
           "-I", CSRC, str(d / "t.cu"), str(d / "stubs.c"), "-o", str(d / "t.so")]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    return C.CDLL(str(d / "t.so"), mode=os.RTLD_LAZY)


def test_limit_is_one_value_for_every_launch_and_not_remembered(fake):
    # two threads launch one kernel with different sizes: neither may leave a limit below the other's need
    assert fake.limit_after_a_launch() == 227 * 1024
    fake.rebuild_context()  # the limit went with the context
    assert fake.limit_after_a_launch() == 227 * 1024
    assert fake.times_asked() == 2
