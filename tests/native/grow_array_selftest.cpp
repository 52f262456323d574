// Host check of GrowArray (cuda_b200/csrc/grow_array.h): what a failed allocation leaves behind.
#include <cstdio>
#include <cstdlib>
#include <set>
#include "../../cuda_b200/csrc/grow_array.h"

static int fails = 0;
#define CHECK(c) \
  do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); fails++; } } while (0)

int main() {
  std::set<void*> live;
  bool full = false;
  auto alloc = [&](void** p, size_t bytes) {
    if (full) return 2;  // as cudaMalloc: *p is not written
    *p = std::malloc(bytes);
    live.insert(*p);
    return 0;
  };
  auto release = [&](void* p) {
    CHECK(live.erase(p) == 1);
    std::free(p);
  };
  lnt::GrowArray<double> a;
  CHECK(a.reserve(0, alloc, release) == 0 && !a.data && !a.cap);
  CHECK(a.reserve(10, alloc, release) == 0 && a.cap == 10 && live.count(a.data));
  double* first = a.data;
  CHECK(a.reserve(7, alloc, release) == 0 && a.data == first);
  CHECK(a.reserve(11, alloc, release) == 0 && a.cap == 20 && live.count(a.data) && live.size() == 1);
  full = true;
  CHECK(a.reserve(20, alloc, release) == 0);
  CHECK(a.reserve(21, alloc, release) == 2 && !a.data && !a.cap && live.empty());
  CHECK(a.reserve(5, alloc, release) == 2 && !a.data && !a.cap);  // not taken for held
  full = false;
  CHECK(a.reserve(5, alloc, release) == 0 && a.cap == 5 && live.count(a.data));
  a.clear(release);
  a.clear(release);
  CHECK(live.empty() && !a.data && !a.cap);
  std::printf(fails ? "FAILED\n" : "ok\n");
  return fails != 0;
}
