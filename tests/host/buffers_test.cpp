// Named device buffers under failing allocations (csrc/buffers.cu against the stand-in runtime).
#include "fake_runtime.hpp"

#include "../../pcaone_b200/csrc/internal.hpp"
#include "../../pcaone_b200/csrc/linalg.hpp"

template <typename F>
bool fails(F&& f) {
  try {
    f();
  } catch (const pg::Error&) {
    return true;
  }
  return false;
}

int main() {
  pcaone_ctx c;
  // the ticket's buffer cannot be allocated, then can: it is cleared before it is used
  fake::malloc_.fail = 1;
  CHECK(fails([&] { pg::tall_counter(&c); }));
  CHECK(*pg::tall_counter(&c) == 0);
  // once: later calls do not clear a running ticket
  *pg::tall_counter(&c) = 5;
  CHECK(*pg::tall_counter(&c) == 5);
  // allocated, but the clearing fails: cleared by the next call
  pg::free_scratch(&c);
  fake::memset_.fail = 1;
  CHECK(fails([&] { pg::tall_counter(&c); }));
  CHECK(*pg::tall_counter(&c) == 0);
  // a buffer whose growth failed is allocated by the next call
  CHECK(pg::scratch(&c, "a", 1000));
  fake::malloc_.fail = 1;
  CHECK(fails([&] { pg::scratch(&c, "a", 2000); }));
  CHECK(pg::scratch(&c, "a", 500));
  pg::free_scratch(&c);
  return 0;
}
