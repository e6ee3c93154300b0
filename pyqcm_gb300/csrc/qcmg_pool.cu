#include "qcmg_pool.h"

#include <cuda.h>

#include <map>
#include <mutex>
#include <vector>

namespace qcmg {

namespace {

struct Lists {
  std::multimap<size_t, void*> dev, pinned;
  size_t dev_bytes = 0, pinned_bytes = 0;
  unsigned long long ctx = 0;
  struct Lane {
    cudaStream_t s;
    cudaEvent_t e[2];
  };
  std::vector<Lane> lanes;
};
constexpr size_t kLanes = 64;  // streams kept

std::mutex g_mu;
// never destroyed: handles may outlive static objects at the process's end
std::map<int, Lists>& lists() {
  static auto* m = new std::map<int, Lists>;
  return *m;
}

int device() {
  int d = 0;
  QCMG_CUDA(cudaGetDevice(&d));
  return d;
}

}  // namespace

unsigned long long context_id() {
  typedef CUresult (*Fn)(CUcontext, unsigned long long*);
  static Fn fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<Fn>(f);
  }();
  unsigned long long id = 0;
  if (!fn || fn(nullptr, &id) != 0) return 0;
  return id;
}

namespace {

// The device's lists, under g_mu; emptied when they are of another context.
Lists& lists_of(int dev, unsigned long long ctx) {
  Lists& l = lists()[dev];
  if (l.ctx != ctx) {
    l = Lists();
    l.ctx = ctx;
  }
  return l;
}

// Sizes are rounded up so that calls of nearly the same size share blocks:
// to the next power of two below 2 MB, to 2 MB above.
size_t rounded(size_t b) {
  constexpr size_t page = (size_t)2 << 20;
  if (b >= page) return (b + page - 1) / page * page;
  size_t r = 512;
  while (r < b) r *= 2;
  return r;
}

void* take(std::multimap<size_t, void*>& m, size_t& held, size_t want, size_t* got) {
  const auto it = m.lower_bound(want);
  if (it == m.end() || it->first > want + want / 4) return nullptr;
  void* p = it->second;
  *got = it->first;
  held -= it->first;
  m.erase(it);
  return p;
}

// Runs an allocation; when there is no memory, once more with the pool empty.
template <class Alloc>
cudaError_t alloc_or_trim(Alloc&& alloc) {
  cudaError_t e = alloc();
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();  // not the next call's error
    pool_trim();
    e = alloc();
  }
  return e;
}

}  // namespace

cudaError_t device_alloc(void** p, size_t bytes) {
  return alloc_or_trim([&] { return cudaMalloc(p, bytes); });
}

cudaError_t pinned_alloc(void** p, size_t bytes) {
  return alloc_or_trim([&] { return cudaMallocHost(p, bytes); });
}

void pool_trim() {
  std::vector<void*> d, h;
  {
    const int dev = device();
    const unsigned long long ctx = context_id();
    std::lock_guard<std::mutex> lock(g_mu);
    Lists& l = lists_of(dev, ctx);
    for (auto& x : l.dev) d.push_back(x.second);
    for (auto& x : l.pinned) h.push_back(x.second);
    l.dev.clear();
    l.pinned.clear();
    l.dev_bytes = l.pinned_bytes = 0;
  }
  for (void* p : d) cudaFree(p);
  for (void* p : h) cudaFreeHost(p);
}

void* pool_get(size_t bytes, size_t* got) {
  const size_t want = rounded(bytes ? bytes : 1);
  {
    const int dev = device();
    const unsigned long long ctx = context_id();
    std::lock_guard<std::mutex> lock(g_mu);
    Lists& l = lists_of(dev, ctx);
    if (void* p = take(l.dev, l.dev_bytes, want, got)) return p;
  }
  void* p = nullptr;
  QCMG_CUDA(device_alloc(&p, want));
  *got = want;
  return p;
}

void pool_put(void* p, size_t got) {
  if (got <= kPoolBytes / 4) {
    cudaPointerAttributes a;
    int dev = 0;
    // to the list of its device, when that is the current one
    if (cudaPointerGetAttributes(&a, p) == cudaSuccess && cudaGetDevice(&dev) == cudaSuccess &&
        a.device == dev) {
      const unsigned long long ctx = context_id();
      std::lock_guard<std::mutex> lock(g_mu);
      Lists& l = lists_of(dev, ctx);
      if (l.dev_bytes + got <= kPoolBytes) {
        l.dev.emplace(got, p);
        l.dev_bytes += got;
        return;
      }
    } else {
      cudaGetLastError();
    }
  }
  cudaFree(p);
}

void* pinned_get(size_t bytes, size_t* got) {
  const size_t want = rounded(bytes ? bytes : 1);
  {
    const int dev = device();
    const unsigned long long ctx = context_id();
    std::lock_guard<std::mutex> lock(g_mu);
    Lists& l = lists_of(dev, ctx);
    if (void* p = take(l.pinned, l.pinned_bytes, want, got)) return p;
  }
  void* p = nullptr;
  QCMG_CUDA(pinned_alloc(&p, want));
  *got = want;
  return p;
}

void pinned_put(void* p, size_t got) {
  cudaPointerAttributes a;
  int dev = 0;
  if (cudaPointerGetAttributes(&a, p) == cudaSuccess && cudaGetDevice(&dev) == cudaSuccess) {
    const unsigned long long ctx = context_id();
    std::lock_guard<std::mutex> lock(g_mu);
    Lists& l = lists_of(dev, ctx);
    if (l.pinned_bytes + got <= kPinnedBytes) {
      l.pinned.emplace(got, p);
      l.pinned_bytes += got;
      return;
    }
  } else {
    cudaGetLastError();
  }
  cudaFreeHost(p);
}

void PoolStream::open() {
  if (s) return;
  device = qcmg::device();
  ctx = context_id();
  {
    std::lock_guard<std::mutex> lock(g_mu);
    Lists& l = lists_of(device, ctx);
    if (!l.lanes.empty()) {
      s = l.lanes.back().s;
      e[0] = l.lanes.back().e[0];
      e[1] = l.lanes.back().e[1];
      l.lanes.pop_back();
      return;
    }
  }
  QCMG_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
  for (auto& x : e) QCMG_CUDA(cudaEventCreateWithFlags(&x, cudaEventDisableTiming));
}

PoolStream::~PoolStream() {
  if (!s) return;
  const bool ok = cudaStreamSynchronize(s) == cudaSuccess && e[0] && e[1];
  if (ok) {
    std::lock_guard<std::mutex> lock(g_mu);
    Lists& l = lists()[device];
    if (l.ctx == ctx && l.lanes.size() < kLanes) {
      l.lanes.push_back({s, {e[0], e[1]}});
      return;
    }
  }
  for (auto x : e)
    if (x) cudaEventDestroy(x);
  cudaStreamDestroy(s);
}

}  // namespace qcmg
