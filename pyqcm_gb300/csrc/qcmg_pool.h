// Device and page-locked memory kept between calls.
//
// A small sector's solve takes a millisecond, and cudaMalloc / cudaFree /
// cudaMallocHost a tenth of that each; cudaFree also waits for every stream
// of the device, so one host thread's clean-up held up the others' solves.
// PoolBuf and PinnedBuf hand their memory back to a per-device list instead.
// The rule for using them: when one goes out of scope, no work that uses its
// memory is pending on any stream (declare a guard that waits after them).
// The lists hold at most kPoolBytes per device (kPinnedBytes of page-locked
// memory); blocks beyond that, and blocks above a quarter of it, go back to
// the driver at once, and all of them when an allocation of the library finds
// no memory, which is then tried once more. After a device reset (another
// context) the lists are forgotten. Safe for any number
// of threads and streams.
#pragma once

#include <cstddef>

#include "qcmg_internal.h"

namespace qcmg {

constexpr size_t kPoolBytes = (size_t)512 << 20;
constexpr size_t kPinnedBytes = (size_t)8 << 20;

// Number of the current context: another one after a device reset, when the
// addresses of the old one mean nothing (or somebody else's memory).
unsigned long long context_id();

// pool_get, pool_put: qcmg_internal.h; on the current device
void* pinned_get(size_t bytes, size_t* got);
void pinned_put(void* p, size_t got);
cudaError_t pinned_alloc(void** p, size_t bytes);  // cudaMallocHost, as device_alloc
void pool_trim();                            // the current device's lists back to the driver

template <class T>
struct PoolBuf {
  T* p = nullptr;
  size_t got = 0;  // bytes
  PoolBuf() = default;
  PoolBuf(const PoolBuf&) = delete;
  PoolBuf& operator=(const PoolBuf&) = delete;
  ~PoolBuf() { release(); }
  void release() {
    if (p) pool_put(p, got);
    p = nullptr;
    got = 0;
  }
  void alloc(size_t count) {
    if (p && count * sizeof(T) <= got) return;
    release();
    p = static_cast<T*>(pool_get(count * sizeof(T), &got));
  }
  void upload(const T* h, size_t count, cudaStream_t s) {
    alloc(count);
    if (count) QCMG_CUDA(cudaMemcpyAsync(p, h, count * sizeof(T), cudaMemcpyHostToDevice, s));
  }
};

template <class T>
struct PinnedBuf {
  T* p = nullptr;
  size_t got = 0;
  PinnedBuf() = default;
  PinnedBuf(const PinnedBuf&) = delete;
  PinnedBuf& operator=(const PinnedBuf&) = delete;
  ~PinnedBuf() {
    if (p) pinned_put(p, got);
  }
  void alloc(size_t count) {
    if (p && count * sizeof(T) <= got) return;
    if (p) pinned_put(p, got);
    p = nullptr;
    p = static_cast<T*>(pinned_get(count * sizeof(T), &got));
  }
};

// Waits for a stream when the scope is left, by an exception too: declared
// after the buffers whose work the stream holds.
struct Drain {
  cudaStream_t s;
  explicit Drain(cudaStream_t st) : s(st) {}
  Drain(const Drain&) = delete;
  Drain& operator=(const Drain&) = delete;
  ~Drain() { cudaStreamSynchronize(s); }
};

// A non-blocking stream and events of the current device, kept likewise.
struct PoolStream {
  cudaStream_t s = nullptr;
  cudaEvent_t e[2] = {nullptr, nullptr};
  int device = 0;
  unsigned long long ctx = 0;
  PoolStream() = default;
  PoolStream(const PoolStream&) = delete;
  PoolStream& operator=(const PoolStream&) = delete;
  ~PoolStream();  // waits for the stream
  void open();
};

}  // namespace qcmg
