"""The memory pool (pyqcm_gb300/csrc/qcmg_pool.cu) against a fake CUDA runtime
with a small device: an allocation that finds no memory is tried once more
after the pool gave back the idle blocks it keeps, for every kind of buffer of
the library; one that cannot be met is refused with the error it had."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "pyqcm_gb300", "csrc")

DRIVER = r"""
#include <cstdio>
#include <cstdlib>
#include <map>
#include "qcmg_pool.cu"

// the runtime: `limit` bytes of device and of page-locked memory
static size_t limit = 0, used[2] = {0, 0};
static std::map<void*, size_t> blocks[2];
static cudaError_t last = cudaSuccess;
static cudaError_t get(int k, void** p, size_t n) {
  if (used[k] + n > limit) return last = cudaErrorMemoryAllocation;
  *p = std::malloc(16);
  blocks[k][*p] = n;
  used[k] += n;
  return cudaSuccess;
}
static cudaError_t put(int k, void* p) {
  used[k] -= blocks[k].at(p);
  blocks[k].erase(p);
  std::free(p);
  return cudaSuccess;
}
extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) { return get(0, p, n); }
cudaError_t cudaMallocHost(void** p, size_t n) { return get(1, p, n); }
cudaError_t cudaFree(void* p) { return put(0, p); }
cudaError_t cudaFreeHost(void* p) { return put(1, p); }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) { return a->device = 0, cudaSuccess; }
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void**, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult*) {
  return cudaErrorNotSupported;
}
cudaError_t cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t*, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t*, unsigned) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
}

using namespace qcmg;
constexpr size_t MB = (size_t)1 << 20;

// `idle` MB in the pool of a device of `total`; `want` MB in a buffer of type B
template <class B>
static int code(size_t total, size_t idle, size_t want) {
  limit = total * MB;
  pool_trim();
  {
    PoolBuf<char> a;
    a.alloc(idle * MB);
    PinnedBuf<char> h;
    h.alloc(idle * MB);
  }
  int r = 0;
  try {
    B b;
    b.alloc(want * MB);
    if (!b.p) r = 100;
  } catch (const Error& e) {
    r = e.code;
    cudaGetLastError();
  }
  if (last != cudaSuccess) r += 1000;  // left for the next call to trip over
  return r;
}
struct Pooled : DevBuf<char> {
  Pooled() { pooled = true; }
};
struct Host {  // page-locked, not from the pool
  void* p = nullptr;
  void alloc(size_t n) { QCMG_CUDA(pinned_alloc(&p, n)); }
  ~Host() {
    if (p) cudaFreeHost(p);
  }
};
template <class B>
static void all() {
  std::printf("%d %d %d %d\n", code<B>(16, 4, 8), code<B>(16, 8, 12), code<B>(16, 8, 16), code<B>(16, 8, 18));
}
int main() {
  all<DevBuf<char>>();
  all<Pooled>();
  all<PoolBuf<char>>();
  all<PinnedBuf<char>>();
  all<Host>();
  pool_trim();
  std::printf("%zu %zu\n", used[0], used[1]);
}
"""


def test_idle_blocks_are_given_back_before_an_allocation_is_refused(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    cuda = "/usr/local/cuda/include"
    if cxx is None or not os.path.exists(os.path.join(cuda, "cuda_runtime.h")):
        pytest.skip("no host C++ compiler or CUDA headers")
    (tmp_path / "driver.cpp").write_text(DRIVER)
    exe = str(tmp_path / "driver")
    subprocess.run([cxx, "-O1", "-std=c++17", "-pthread", "-I", cuda, "-I", CSRC, "-I", os.path.join(ROOT, "include"),
                    str(tmp_path / "driver.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, check=True).stdout.splitlines()
    # fits beside the idle blocks, in their place, in all there is; does not fit (QCMG_ERR_NOMEM = -3)
    assert out[:5] == ["0 0 0 -3"] * 5
    assert out[5] == "0 0"
