// Device and pinned host memory of the library's short-lived objects.
//
// A run, an input schedule or an e-prop minibatch lives for one call of a
// user's loop; on a B200 cudaMalloc + cudaFree of its buffers took 1.4 ms of a
// 2.1 ms minibatch (784-256-10 net, 64 samples) and cudaHostAlloc of a result
// block 2.5 ms, as long as the work itself.  Released blocks are therefore
// kept, by size class and device, and handed out again.
//
//   safe      a block is taken back only after the wait that cudaFree makes for
//             its device, so no stream of any thread can still use it; one mutex
//             guards the lists
//   bounded   at most kKeepDevice bytes per device and kKeepHost pinned bytes
//             are kept; a block that would exceed them is freed, and one that
//             never could be kept is not rounded up to a class
//   returned  everything kept is freed when the last live block is released
//             and when an allocation fails (which is then tried again, without
//             the rounding)
#include <map>
#include <mutex>
#include <unordered_map>
#include <utility>
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

// Two small allocations of a device: `spare` is freed to wait for the device and
// allocated again; `anchor` keeps the driver's page of small blocks mapped
// meanwhile (mapping one takes hundreds of microseconds).
struct Token {
  void *anchor = nullptr, *spare = nullptr;
};

struct Pool {
  std::mutex mu;
  std::unordered_map<void*, Block> live;
  std::map<std::pair<int, size_t>, std::vector<void*>> kept;
  std::map<int, size_t> kept_bytes;
  std::map<int, Token> tokens;
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

// Calls in its scope do not disturb a stream capture of any thread, nor does a
// capture forbid them.
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// Waits for all work of the current device `dev`, on every stream, the way
// releasing a block without a pool did: by cudaFree, of a small block.
// cudaDeviceSynchronize would wait alike, but invalidates any stream capture
// under way in another thread (this library's own of a run, or a framework's).
// 4.1 us on an idle device against 3.3.
bool wait_device(Pool& q, int dev) {
  void *first = nullptr, *next = nullptr;
  bool anchored;
  {
    std::lock_guard<std::mutex> lk(q.mu);
    Token& t = q.tokens[dev];
    anchored = t.anchor != nullptr;
    std::swap(first, t.spare);
  }
  void* anchor = nullptr;
  if (!anchored && cudaMalloc(&anchor, 1) != cudaSuccess) anchor = nullptr;
  if (!first && cudaMalloc(&first, 1) != cudaSuccess) first = nullptr;
  const bool ok = first && cudaFree(first) == cudaSuccess;
  if (ok && cudaMalloc(&next, 1) != cudaSuccess) next = nullptr;
  {
    std::lock_guard<std::mutex> lk(q.mu);
    Token& t = q.tokens[dev];
    if (!t.anchor) std::swap(anchor, t.anchor);
    if (!t.spare) std::swap(next, t.spare);
  }
  if (anchor) cudaFree(anchor);
  if (next) cudaFree(next);
  return ok;
}

// Takes back blocks, after one wait for each of their devices: nothing that was
// launched before this call may still use them.
void give_back(const std::vector<void*>& ps) {
  if (ps.empty()) return;
  Pool& q = pool();
  std::vector<std::pair<void*, Block>> bs;
  {
    std::lock_guard<std::mutex> lk(q.mu);
    for (void* p : ps) {
      auto it = q.live.find(p);
      if (it != q.live.end()) bs.push_back(*it);
    }
  }
  const RelaxedCapture relaxed;
  int cur = 0;
  const bool known = cudaGetDevice(&cur) == cudaSuccess;
  std::map<int, bool> idle;  // by Block::dev
  for (const auto& b : bs) {
    const int dev = b.second.dev;
    if (!known || idle.count(dev)) continue;
    const bool sw = dev != kHost && cur != dev;
    if (sw) cudaSetDevice(dev);
    idle[dev] = wait_device(q, sw ? dev : cur);
    if (sw) cudaSetDevice(cur);
  }
  std::lock_guard<std::mutex> lk(q.mu);
  for (const auto& pb : bs) {
    const Block& b = pb.second;
    q.live.erase(pb.first);
    size_t& kept = q.kept_bytes[b.dev];
    if (idle[b.dev] && b.classed && kept + b.bytes <= keep_limit(b.dev)) {
      q.kept[{b.dev, b.bytes}].push_back(pb.first);
      kept += b.bytes;
    } else {
      raw_free(pb.first, b.dev);
      cudaGetLastError();
    }
  }
  if (q.live.empty()) {
    for (auto& k : q.kept_bytes) trim(q, k.first);
    for (auto& t : q.tokens) {
      if (t.second.anchor) cudaFree(t.second.anchor);
      if (t.second.spare) cudaFree(t.second.spare);
      t.second = Token();
    }
  }
}

// Blocks that this thread releases within a PoolBatch.
thread_local int later_depth = 0;
thread_local std::vector<void*> later;

int take(void** out, size_t n, int dev) {
  size_t c = size_class(n, dev);
  Pool& q = pool();
  std::unique_lock<std::mutex> lk(q.mu);
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
      lk.unlock();
      give_back(std::exchange(later, {}));
      lk.lock();
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
  if (later_depth) later.push_back(p);
  else give_back({p});
}

PoolBatch::PoolBatch() { ++later_depth; }

PoolBatch::~PoolBatch() {
  if (--later_depth == 0) give_back(std::exchange(later, {}));
}

}  // namespace sncb
