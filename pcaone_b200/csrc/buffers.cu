// Named device buffers of a context (host code only).
#include <algorithm>

#include "internal.hpp"
#include "linalg.hpp"

namespace pg {

void* scratch(pcaone_ctx* c, const std::string& name, size_t bytes) {
  DevBuf& b = c->bufs[name];
  if (b.bytes < bytes) {
    if (b.p) PG_CUDA(cudaFree(b.p));
    b.p = nullptr;
    b.bytes = 0;
    size_t alloc = round_up(std::max<size_t>(bytes, 256), 256);
    PG_CUDA(cudaMalloc(&b.p, alloc));
    b.bytes = alloc;
  }
  return b.p;
}

void free_scratch(pcaone_ctx* c) {
  for (auto& kv : c->bufs)
    if (kv.second.p) cudaFree(kv.second.p);
  c->bufs.clear();
  c->tall_ticket_zero = false;
}

unsigned* tall_counter(pcaone_ctx* c) {
  unsigned* p = (unsigned*)scratch(c, "tall_cnt", sizeof(unsigned));
  if (!c->tall_ticket_zero) {  // cleared once its first clearing is queued, whatever failed before
    PG_CUDA(cudaMemsetAsync(p, 0, sizeof(unsigned), c->stream));
    c->tall_ticket_zero = true;
  }
  return p;
}

}  // namespace pg
