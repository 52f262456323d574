// A device array that only grows, for descriptors uploaded before a launch.
#pragma once
#include <algorithm>
#include <cstddef>

namespace lnt {

template <class T>
struct GrowArray {
  T* data = nullptr;
  size_t cap = 0;  // elements that `data` holds

  // Room for `want` elements; the contents are not kept.  alloc(void** p, bytes) returns 0 on success.
  // After a failure the array is empty, so the next call tries again.
  template <class Alloc, class Free>
  auto reserve(size_t want, Alloc alloc, Free release) -> decltype(alloc((void**)nullptr, (size_t)0)) {
    using Status = decltype(alloc((void**)nullptr, (size_t)0));
    if (want <= cap) return Status(0);
    const size_t next = std::max(want, 2 * cap);
    clear(release);
    void* p = nullptr;
    const Status st = alloc(&p, next * sizeof(T));
    if (st == Status(0)) {
      data = (T*)p;
      cap = next;
    }
    return st;
  }
  template <class Free>
  void clear(Free release) {
    if (data) release(data);
    data = nullptr;
    cap = 0;
  }
};

}  // namespace lnt
