// Device and pinned host memory of the library's short-lived objects.
//
// A run, an input schedule or an e-prop minibatch lives for one call of a
// user's loop; on a B200 cudaMalloc + cudaFree of its buffers took 1.4 ms of a
// 2.1 ms minibatch (784-256-10 net, 64 samples) and cudaHostAlloc of a result
// block 2.5 ms, as long as the work itself.  Released blocks are therefore
// kept, by size class and device, and handed out again.
//
//   safe      a block is taken back only after cudaDeviceSynchronize on its
//             device -- the wait cudaFree makes as well -- so no stream of any
//             thread can still use it; one mutex guards the lists
//   bounded   at most kKeepDevice bytes per device and kKeepHost pinned bytes
//             are kept; a block that would exceed them is freed, and one that
//             never could be kept is not rounded up to a class
//   returned  everything kept is freed when the last live block is released
//             and when an allocation fails (which is then tried again, without
//             the rounding)
#include <map>
#include <mutex>
#include <unordered_map>
#include <vector>

#include "internal.h"

namespace sncb {

namespace {

constexpr size_t kKeepDevice = size_t(256) << 20;
constexpr size_t kKeepHost = size_t(32) << 20;
constexpr int kHost = -1;  // "device" of pinned host blocks

size_t keep_limit(int dev) { return dev == kHost ? kKeepHost : kKeepDevice; }

struct Block {
  int dev;
  size_t bytes;
  bool classed;  // its size is a class, so another allocation can take it
};

struct Pool {
  std::mutex mu;
  std::unordered_map<void*, Block> live;
  std::map<std::pair<int, size_t>, std::vector<void*>> kept;
  std::map<int, size_t> kept_bytes;
};

// Never destroyed: objects may be released while the process exits.
Pool& pool() {
  static Pool* p = new Pool();
  return *p;
}

// Powers of two up to 1 MiB, then four sizes between each two; blocks too large
// to be kept as they are.
size_t size_class(size_t n, int dev) {
  if (n > keep_limit(dev)) return n;
  size_t c = 512;
  while (c < n) c <<= 1;
  if (c > (size_t(1) << 20)) {
    const size_t step = c >> 3;  // c / 2 < n <= c
    c = (n + step - 1) / step * step;
  }
  return c;
}

cudaError_t raw_alloc(void** p, size_t n, int dev) {
  return dev == kHost ? cudaHostAlloc(p, n, cudaHostAllocDefault) : cudaMalloc(p, n);
}

void raw_free(void* p, int dev) {
  if (dev == kHost) cudaFreeHost(p);
  else cudaFree(p);
}

// Frees every kept block of `dev` (kHost: the pinned ones).
void trim(Pool& q, int dev) {
  for (auto& k : q.kept)
    if (k.first.first == dev) {
      for (void* p : k.second) raw_free(p, dev);
      k.second.clear();
    }
  q.kept_bytes[dev] = 0;
}

int take(void** out, size_t n, int dev) {
  size_t c = size_class(n, dev);
  Pool& q = pool();
  std::lock_guard<std::mutex> lk(q.mu);
  auto& list = q.kept[{dev, c}];
  void* p = nullptr;
  if (!list.empty()) {
    p = list.back();
    list.pop_back();
    q.kept_bytes[dev] -= c;
  } else {
    cudaError_t e = raw_alloc(&p, c, dev);
    if (e == cudaErrorMemoryAllocation) {
      cudaGetLastError();
      trim(q, dev);
      c = n;  // what was asked for is what must fit
      e = raw_alloc(&p, c, dev);
    }
    if (e != cudaSuccess) return cuda_fail(e, dev == kHost ? "cudaHostAlloc" : "cudaMalloc");
  }
  q.live[p] = Block{dev, c, c == size_class(n, dev)};
  *out = p;
  return SNC_B200_OK;
}

}  // namespace

int pool_alloc(void** p, size_t n) {
  *p = nullptr;
  if (alloc_fault()) { set_error("device allocation failed (injected)"); return SNC_B200_ENOMEM; }
  int dev = 0;
  SNCB_CUDA(cudaGetDevice(&dev));
  return take(p, n, dev);
}

int pool_alloc_host(void** p, size_t n) {
  *p = nullptr;
  return take(p, n, kHost);
}

void pool_free(void* p) {
  if (!p) return;
  Pool& q = pool();
  Block b;
  {
    std::lock_guard<std::mutex> lk(q.mu);
    auto it = q.live.find(p);
    if (it == q.live.end()) return;
    b = it->second;
  }
  // nothing that was launched before this call may still use the block
  int cur = 0;
  const bool sw = b.dev != kHost && cudaGetDevice(&cur) == cudaSuccess && cur != b.dev;
  if (sw) cudaSetDevice(b.dev);
  const bool idle = cudaDeviceSynchronize() == cudaSuccess;
  std::lock_guard<std::mutex> lk(q.mu);
  q.live.erase(p);
  size_t& kept = q.kept_bytes[b.dev];
  if (idle && b.classed && kept + b.bytes <= keep_limit(b.dev)) {
    q.kept[{b.dev, b.bytes}].push_back(p);
    kept += b.bytes;
  } else {
    raw_free(p, b.dev);
    cudaGetLastError();
  }
  if (q.live.empty())
    for (auto& k : q.kept_bytes) trim(q, k.first);
  if (sw) cudaSetDevice(cur);
}

}  // namespace sncb
