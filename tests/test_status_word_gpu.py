"""The library-wide status word: kernels and CTAs that report at the same moment all leave their bit (raise_status of
csrc/common.cuh, on a word in mapped host memory as csrc/capi.cu allocates it)."""
import ctypes
import os
import subprocess

import pytest

from exact_b200 import _build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "common.cuh"
__global__ void raise_all(int* word) { if (threadIdx.x == 0) exb::raise_status(word, 1 << (blockIdx.x % 31)); }
extern "C" __attribute__((visibility("default"))) int raised(int streams, int blocks) {
  int* word = nullptr;
  if (cudaHostAlloc((void**)&word, 64, cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) return -1;
  *word = 0;
  cudaStream_t st[4];
  for (int i = 0; i < streams; i++) cudaStreamCreateWithFlags(&st[i], cudaStreamNonBlocking);
  for (int i = 0; i < streams; i++) raise_all<<<blocks, 32, 0, st[i]>>>(word);
  int out = cudaDeviceSynchronize() == cudaSuccess ? *(volatile int*)word : -1;
  for (int i = 0; i < streams; i++) cudaStreamDestroy(st[i]);
  cudaFreeHost(word);
  return out;
}
"""


def test_concurrent_reports_lose_no_bit(tmp_path):
    src, lib = tmp_path / "raise.cu", str(tmp_path / "raise.so")
    src.write_text(SOURCE)
    subprocess.run([_build._nvcc()] + _build.NVCC_FLAGS + ["-shared", str(src), "-o", lib], check=True, cwd=os.path.dirname(_build.PKG))
    raised = ctypes.CDLL(lib).raised
    for _ in range(50):
        assert raised(4, 31 * 20) == (1 << 31) - 1
