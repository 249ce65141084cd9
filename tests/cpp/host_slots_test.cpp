// HostSlots (libbi_b200/csrc/host_slots.h) with a fake allocator.
#include "../../libbi_b200/csrc/host_slots.h"

#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <set>
#include <thread>
#include <vector>

static int allocs = 0;
static bool fail = false, gone = false;
static void* fake_alloc(size_t bytes) {
  if (fail) return nullptr;
  ++allocs;
  gone = false;
  return std::calloc(1, bytes);
}
static bool fake_valid(void*) { return !gone; }

#define CHECK(c)                                       \
  do {                                                 \
    if (!(c)) {                                        \
      std::printf("line %d: %s\n", __LINE__, #c);      \
      return 1;                                        \
    }                                                  \
  } while (0)

int main() {
  typedef bpf::HostSlots<long long, 8> Slots;
  {  // short-lived handles, one after another: one allocation
    Slots s(fake_alloc, fake_valid);
    for (int i = 0; i < 100; ++i) {
      long long* p = s.acquire();
      CHECK(p);
      s.release(p);
    }
    CHECK(allocs == 1);
    // a block that went is replaced, also while a slot of it is held
    gone = true;
    long long* p = s.acquire();
    CHECK(p && allocs == 2);
    gone = true;
    long long* q = s.acquire();
    CHECK(q && q != p && allocs == 3);
    s.release(p);
    for (int i = 0; i < 7; ++i) CHECK(s.acquire());
    CHECK(!s.acquire());
  }
  {  // distinct slots, none left after the last, one again after a release
    Slots s(fake_alloc, fake_valid);
    std::set<long long*> held;
    for (int i = 0; i < 8; ++i) held.insert(s.acquire());
    CHECK(held.size() == 8 && !held.count(nullptr));
    CHECK(!s.acquire());
    s.release(nullptr);
    s.release(*held.begin());
    CHECK(s.acquire() == *held.begin());
    CHECK(allocs == 4);
  }
  {  // no pinned memory: no slot, and a later try may succeed
    Slots s(fake_alloc, fake_valid);
    fail = true;
    CHECK(!s.acquire());
    fail = false;
    CHECK(s.acquire());
  }
  {  // threads never share a slot
    Slots s(fake_alloc, fake_valid);
    std::atomic<int> clashes(0), got(0);
    std::vector<std::thread> ts;
    for (int t = 0; t < 16; ++t)
      ts.emplace_back([&, t] {
        for (int i = 0; i < 20000; ++i) {
          long long* p = s.acquire();
          if (!p) continue;
          ++got;
          *(volatile long long*)p = t;
          std::this_thread::yield();
          if (*(volatile long long*)p != t) ++clashes;
          s.release(p);
        }
      });
    for (std::thread& t : ts) t.join();
    CHECK(clashes == 0 && got > 0);
  }
  std::puts("ok");
  return 0;
}
