// Copies of pageable host memory. The runtime moves it through one staging buffer with one host
// thread, and a large fresh result array is faulted in page by page on the way. A few threads that each
// copy 1 MiB chunks between the caller's array and a pinned slot keep the link and the page faults
// going together. Whole calls, with 16 host cores, two and one (through the runtime: 28, 56 and 2.0 ms):
// a load of 100 MB of records 3.5, 7.0 and 12.4 ms; an LD call with 256 MB of results 17, 41 and 56 ms, with
// 10 MB 1.6, 1.4 and 1.9.
// Sets of slots (8 MiB each) are kept in the process and shared by its contexts: a copy takes a set of its
// own, at most two idle sets are kept, and the last context's end frees them. Streams belong to
// the context; the threads live for one call.
// Pinning a set takes 3 to 11 ms, so it is pinned once the copies that a context made without one come
// to kXferPaidOff (first LD call of a context, 2504 x 5000 with 10 MB of results: 1.6 to 3 ms;
// 10 to 16 with a set pinned at once). Where a set cannot be had the runtime's path serves, and
// memory that the caller has pinned goes straight to the link (a load of 100 MB of records: 1.9 ms;
// through the slots 3.5 with 16 host cores, 12.4 with one).
#include "xfer.hpp"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

namespace pg {

namespace {
constexpr int kMaxWorkers = 8;
constexpr size_t kKeptSets = 2;

struct SlotPool {
  std::mutex mu;
  std::vector<void*> idle;
  int contexts = 0;
};
SlotPool& pool() {
  static SlotPool* p = new SlotPool;  // never destroyed: contexts may outlive static destructors
  return *p;
}

void* idle_set() {
  std::lock_guard<std::mutex> g(pool().mu);
  if (pool().idle.empty()) return nullptr;
  void* p = pool().idle.back();
  pool().idle.pop_back();
  return p;
}

// Whether the device reaches host memory [p, p + bytes) by itself (pinned by the caller).
bool reachable(const void* p, size_t bytes) {
  cudaPointerAttributes a{}, b{};
  const bool ok = cudaPointerGetAttributes(&a, p) == cudaSuccess &&
                  cudaPointerGetAttributes(&b, (const char*)p + bytes - 1) == cudaSuccess;
  if (!ok) (void)cudaGetLastError();
  return ok && a.type != cudaMemoryTypeUnregistered && b.type != cudaMemoryTypeUnregistered;
}
}  // namespace

XferSlots::~XferSlots() {
  if (!p_) return;
  {
    std::lock_guard<std::mutex> g(pool().mu);
    if (pool().contexts > 0 && pool().idle.size() < kKeptSets) {
      pool().idle.push_back(p_);
      return;
    }
  }
  cudaFreeHost(p_);
}

XferSlots xfer_slots(pcaone_ctx* c, const void* host, size_t bytes) {
  if (bytes < kXferMin || reachable(host, bytes)) return XferSlots(nullptr);
  void* p = idle_set();
  if (!p) {
    c->xfer_paged += bytes;
    if (c->xfer_paged < kXferPaidOff) return XferSlots(nullptr);
    if (cudaHostAlloc(&p, (size_t)xfer_workers() * kXferSlot, cudaHostAllocPortable) != cudaSuccess) {
      (void)cudaGetLastError();
      return XferSlots(nullptr);
    }
  }
  XferSlots slots(p);
  c->xfer_streams.resize(xfer_workers(), nullptr);
  for (cudaStream_t& s : c->xfer_streams)
    if (!s && cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess) {
      (void)cudaGetLastError();
      s = nullptr;
      return XferSlots(nullptr);
    }
  return slots;
}

int xfer_workers() {
  return (int)std::max(1u, std::min((unsigned)kMaxWorkers, std::thread::hardware_concurrency()));
}

void xfer_chunks(pcaone_ctx* c, const XferSlots& slots, int64_t chunks, const XferChunk& f) {
  const int workers = (int)std::min<int64_t>(xfer_workers(), chunks);
  PG_CUDA(cudaStreamSynchronize(c->stream));
  std::atomic<int64_t> next{0};
  std::mutex mu;
  int code = PCAONE_OK;
  std::string what;
  auto work = [&](int t) {
    try {
      PG_CUDA(cudaSetDevice(c->device));
      for (int64_t i; (i = next.fetch_add(1)) < chunks;) {
        f(i, t, slots.slot(t), c->xfer_streams[t]);
        PG_CUDA(cudaStreamSynchronize(c->xfer_streams[t]));
      }
    } catch (const Error& e) {
      next = chunks;
      std::lock_guard<std::mutex> g(mu);
      if (code == PCAONE_OK) {
        code = e.code;
        what = e.what();
      }
    } catch (const std::exception& e) {
      next = chunks;
      std::lock_guard<std::mutex> g(mu);
      if (code == PCAONE_OK) {
        code = PCAONE_ECUDA;
        what = e.what();
      }
    }
  };
  std::vector<std::thread> th;
  th.reserve(workers);
  try {
    for (int t = 1; t < workers; ++t) th.emplace_back(work, t);
  } catch (...) {  // no more threads: go on with those there are
  }
  work(0);
  for (auto& x : th) x.join();
  if (code != PCAONE_OK) {
    for (auto s : c->xfer_streams)  // nothing may still use the slots or the caller's buffers
      if (s) cudaStreamSynchronize(s);
    throw Error(code, what);
  }
}

namespace {
// The runtime's own path.
void copy_plain(pcaone_ctx* c, void* dst, const void* src, size_t bytes, cudaMemcpyKind kind) {
  if (bytes) PG_CUDA(cudaMemcpyAsync(dst, src, bytes, kind, c->stream));
  PG_CUDA(cudaStreamSynchronize(c->stream));
}
int64_t chunks_of(size_t bytes) { return (int64_t)((bytes + kXferSlot - 1) / kXferSlot); }
}  // namespace

void copy_to_host(pcaone_ctx* c, void* dst, const void* src, size_t bytes) {
  const XferSlots slots = xfer_slots(c, dst, bytes);
  if (!slots) return copy_plain(c, dst, src, bytes, cudaMemcpyDeviceToHost);
  xfer_chunks(c, slots, chunks_of(bytes), [&](int64_t i, int, char* slot, cudaStream_t st) {
    const size_t o = (size_t)i * kXferSlot, n = std::min(kXferSlot, bytes - o);
    PG_CUDA(cudaMemcpyAsync(slot, (const char*)src + o, n, cudaMemcpyDeviceToHost, st));
    PG_CUDA(cudaStreamSynchronize(st));
    std::memcpy((char*)dst + o, slot, n);
  });
}

void copy_to_device(pcaone_ctx* c, void* dst, const void* src, size_t bytes) {
  const XferSlots slots = xfer_slots(c, src, bytes);
  if (!slots) return copy_plain(c, dst, src, bytes, cudaMemcpyHostToDevice);
  xfer_chunks(c, slots, chunks_of(bytes), [&](int64_t i, int, char* slot, cudaStream_t st) {
    const size_t o = (size_t)i * kXferSlot, n = std::min(kXferSlot, bytes - o);
    std::memcpy(slot, (const char*)src + o, n);
    PG_CUDA(cudaMemcpyAsync((char*)dst + o, slot, n, cudaMemcpyHostToDevice, st));
  });
}

void xfer_open(pcaone_ctx*) {
  std::lock_guard<std::mutex> g(pool().mu);
  ++pool().contexts;
}

void xfer_close(pcaone_ctx* c) {
  for (auto s : c->xfer_streams)
    if (s) {
      cudaStreamSynchronize(s);
      cudaStreamDestroy(s);
    }
  c->xfer_streams.clear();
  std::vector<void*> gone;
  {
    std::lock_guard<std::mutex> g(pool().mu);
    if (--pool().contexts == 0) gone.swap(pool().idle);
  }
  for (void* p : gone) cudaFreeHost(p);
}

}  // namespace pg
