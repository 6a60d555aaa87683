// Large host copies (csrc/xfer.cu against the stand-in runtime): their path, and that every byte arrives
// on each of them.
#include "fake_runtime.hpp"

#include <string>
#include <thread>
#include <vector>

#include "../../pcaone_b200/csrc/xfer.hpp"

namespace {
constexpr size_t MiB = size_t(1) << 20;

std::vector<char> bytes(size_t n, unsigned seed) {
  std::vector<char> v(n);
  for (size_t i = 0; i < n; ++i) v[i] = (char)((i * 2654435761u + seed) >> 7);
  return v;
}

struct Context : pcaone_ctx {
  Context() { pg::xfer_open(this); }
  ~Context() { pg::xfer_close(this); }
};

// Copies n bytes to the "device" and back; every byte arrives and no error is left behind.
void round_trip(pcaone_ctx* c, size_t n, unsigned seed = 1) {
  const std::vector<char> in = bytes(n, seed);
  std::vector<char> dev(n), out(n);
  pg::copy_to_device(c, dev.data(), in.data(), n);
  CHECK(dev == in);
  pg::copy_to_host(c, out.data(), dev.data(), n);
  CHECK(out == in);
  CHECK(!fake::error_left);
}

// Calls that f makes of one kind.
template <typename F>
int calls(const fake::Call& k, F&& f) {
  const int before = k.calls;
  f();
  return k.calls - before;
}

void small_and_cold_copies_take_one_call() {
  Context c;
  const std::vector<char> in = bytes(10 * MiB, 3);
  std::vector<char> dev(in.size());
  auto copy = [&](size_t n) { pg::copy_to_device(&c, dev.data(), in.data(), n); };
  CHECK(calls(fake::host_alloc, [&] {
          for (const size_t n : {size_t(0), size_t(1), 8 * MiB - 1})
            CHECK(calls(fake::copy, [&] { copy(n); }) == (n ? 1 : 0));
          for (int i = 0; i < 3; ++i) CHECK(calls(fake::copy, [&] { copy(10 * MiB); }) == 1);  // 30 MiB in all
        }) == 0);
  CHECK(calls(fake::host_alloc, [&] { CHECK(calls(fake::copy, [&] { copy(10 * MiB); }) == 10); }) == 1);  // paid off
  CHECK(calls(fake::host_alloc, [&] { CHECK(calls(fake::copy, [&] { copy(9 * MiB + 5); }) == 10); }) == 0);
  CHECK(dev == in);
}

void large_copies_pin_a_set_once() {
  {
    Context c;
    CHECK(calls(fake::host_alloc, [&] {
            round_trip(&c, 40 * MiB + 12345);
            round_trip(&c, 33 * MiB, 7);
          }) == 1);
    Context d;  // the idle set serves another context, whatever that one has copied
    CHECK(calls(fake::host_alloc, [&] { round_trip(&d, 8 * MiB); }) == 0);
  }
  CHECK(fake::host_free.calls == fake::host_alloc.calls);
}

void copies_go_on_without_slots() {
  Context c;
  fake::host_alloc.fail = 1;
  round_trip(&c, 40 * MiB);
  fake::host_alloc.fail = 1000000;
  for (int i = 0; i < 3; ++i) round_trip(&c, 33 * MiB + i);
  fake::host_alloc.fail = 0;
  for (int failing = 1; failing <= 3; ++failing) {  // some of the streams cannot be had
    Context d;
    fake::stream_create.fail = failing;
    round_trip(&d, 40 * MiB);
    round_trip(&d, 40 * MiB);
    CHECK(fake::stream_create.fail == 0);
  }
  CHECK(calls(fake::copy, [&] { round_trip(&c, 40 * MiB); }) == 80);
}

void pinned_memory_is_not_staged() {
  Context c;
  round_trip(&c, 40 * MiB);
  const std::vector<char> in = bytes(40 * MiB, 5);
  std::vector<char> dev(in.size()), out(in.size());
  fake::pinned_from = in.data();
  fake::pinned_to = in.data() + in.size();
  CHECK(calls(fake::copy, [&] { pg::copy_to_device(&c, dev.data(), in.data(), in.size()); }) == 1);
  fake::pinned_from = out.data();
  fake::pinned_to = out.data() + out.size();
  CHECK(calls(fake::copy, [&] { pg::copy_to_host(&c, out.data(), dev.data(), out.size()); }) == 1);
  CHECK(out == in);
  fake::pinned_to -= 1;  // the last byte is not
  CHECK(calls(fake::copy, [&] { pg::copy_to_host(&c, out.data(), dev.data(), out.size()); }) == 40);
  fake::pinned_from = fake::pinned_to = nullptr;
}

void failed_copies_leave_the_context_usable() {
  Context c;
  round_trip(&c, 40 * MiB);
  std::vector<char> dev(40 * MiB), out(40 * MiB);
  fake::copy.fail = 1;
  bool failed = false;
  try {
    pg::copy_to_host(&c, out.data(), dev.data(), out.size());
  } catch (const pg::Error& e) {
    failed = e.code == PCAONE_EOOM;
  }
  CHECK(failed);
  fake::error_left = false;
  CHECK(calls(fake::host_alloc, [&] { round_trip(&c, 40 * MiB); }) == 0);
}

void contexts_copy_at_once() {
  {
    Context c[4];
    std::vector<std::thread> th;
    for (int t = 0; t < 4; ++t)
      th.emplace_back([&, t] {
        for (int i = 0; i < 3; ++i) round_trip(&c[t], 33 * MiB + 17 * t, 100 * t + i);
      });
    for (auto& x : th) x.join();
    CHECK(fake::host_alloc.calls - fake::host_free.calls <= 2);  // idle sets kept
  }
  CHECK(fake::host_free.calls == fake::host_alloc.calls);
}
}  // namespace

int main(int argc, char** argv) {
  const std::string name = argc > 1 ? argv[1] : "";
  if (name == "cold") small_and_cold_copies_take_one_call();
  else if (name == "large") large_copies_pin_a_set_once();
  else if (name == "no_slots") copies_go_on_without_slots();
  else if (name == "pinned") pinned_memory_is_not_staged();
  else if (name == "failed") failed_copies_leave_the_context_usable();
  else if (name == "at_once") contexts_copy_at_once();
  else return 2;
  return 0;
}
