"""A bounded wait that runs out: the kernel returns, and its code is in the
page-locked error flag when the stream has been waited for."""
import ctypes
import subprocess

import pytest

from gdpy import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <stdlib.h>
#include <unistd.h>
#include "gd_common.cuh"
#include "gd_ptx.cuh"
__global__ void k(int arrive, int* err) {
  __shared__ uint64_t bar;
  gd::mbar_init(gd::smem_u32(&bar), 1);
  if (arrive) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(gd::smem_u32(&bar)) : "memory");
  gd::mbar_wait(gd::smem_u32(&bar), 0, err, 77);
}
extern "C" int run(int arrive) {
  const size_t page = (size_t)sysconf(_SC_PAGESIZE);
  int *err = (int*)aligned_alloc(page, page), *derr = nullptr;
  cudaStream_t s;
  if (!err || cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess ||
      cudaHostRegister(err, page, cudaHostRegisterMapped) != cudaSuccess ||
      cudaHostGetDevicePointer(&derr, err, 0) != cudaSuccess)
    return -1;
  *err = 0;
  k<<<1, 1, 0, s>>>(arrive, derr);
  const int got = cudaStreamSynchronize(s) == cudaSuccess ? *(volatile int*)err : -1;
  cudaHostUnregister(err);
  free(err);
  cudaStreamDestroy(s);
  return got;
}
"""


def test_flag(tmp_path):
    src, so = str(tmp_path / "w.cu"), str(tmp_path / "w.so")
    open(src, "w").write(SOURCE)
    subprocess.run([build.nvcc(), *build.ARCH, *build.FLAGS, "-shared", src, "-o", so], check=True)
    lib = ctypes.CDLL(so)
    assert lib.run(1) == 0
    assert lib.run(0) == 77
    assert lib.run(1) == 0
