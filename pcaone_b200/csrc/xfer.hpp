// Large copies between pageable host memory and the device (xfer.cu).
#pragma once

#include <functional>

#include "internal.hpp"

namespace pg {

// One chunk of a large copy, run by worker `worker` (each has a pinned slot of kXferSlot bytes and
// a stream of its own); the worker waits for the stream after it.
using XferChunk = std::function<void(int64_t chunk, int worker, char* slot, cudaStream_t stream)>;
constexpr size_t kXferSlot = size_t(1) << 20;
// Copies below this size take the runtime's own path: the workers cost 0.1 to 0.2 ms to start, and it
// still does 17 to 20 GB/s there (4 MB: 0.24 ms against 0.46; 8 MB: 0.45 against 0.38).
constexpr size_t kXferMin = size_t(8) << 20;

// A set of slots is pinned for a context whose copies without one have come to this: they took 0.05
// (recently used pages) to 0.45 ms (fresh ones) a MiB longer, the set takes 3 to 11 ms.
constexpr size_t kXferPaidOff = size_t(32) << 20;

// A set of pinned slots, one a worker, held for the length of a copy.
class XferSlots {
 public:
  explicit XferSlots(void* p) : p_(p) {}
  XferSlots(XferSlots&& o) noexcept : p_(o.p_) { o.p_ = nullptr; }
  XferSlots(const XferSlots&) = delete;
  XferSlots& operator=(const XferSlots&) = delete;
  ~XferSlots();
  explicit operator bool() const { return p_ != nullptr; }
  char* slot(int worker) const { return (char*)p_ + (size_t)worker * kXferSlot; }

 private:
  void* p_;
};

// Slots for a copy of bytes from or to `host`; none where the runtime's own copy serves better (a small
// copy, memory that is pinned already, a set not paid off) or the slots cannot be had.
XferSlots xfer_slots(pcaone_ctx* c, const void* host, size_t bytes);

// Runs f for the chunks 0 .. chunks - 1 on a few host threads, after the work queued on the
// context's stream; returns when all of it is complete.
void xfer_chunks(pcaone_ctx* c, const XferSlots& slots, int64_t chunks, const XferChunk& f);
int xfer_workers();

// Synchronous copies, after the work queued on the context's stream.
void copy_to_host(pcaone_ctx* c, void* dst, const void* src, size_t bytes);
void copy_to_device(pcaone_ctx* c, void* dst, const void* src, size_t bytes);

// Called when a context is created and destroyed: the pinned slots are kept between copies while
// any context of the process lives.
void xfer_open(pcaone_ctx* c);
void xfer_close(pcaone_ctx* c);

}  // namespace pg
