// Growth of the backend's device scratch.  No CUDA in here: the caller brings allocation and release.
#pragma once

#include <algorithm>
#include <cstddef>
#include <vector>

// A buffer that grows on demand.  Once a launch that uses it went into a CUDA graph (`recorded`), the graph holds its
// address and may be replayed as long as the backend lives: growing then keeps the old buffer.
struct tb_scratch {
  void* ptr = nullptr;
  size_t cap = 0;
  bool recorded = false;
};

// Makes `s` hold `need` bytes; false when there is no memory (a recorded buffer is then left as it was).
// A recorded buffer goes to `kept`, and its successor is at least twice as large, so that all that is kept is
// smaller than what is in use.  `alloc(bytes)` returns null on failure, `release(ptr)` frees.
template <class Alloc, class Release>
bool tb_scratch_grow(tb_scratch* s, std::vector<void*>* kept, size_t need, Alloc alloc, Release release) {
  if (s->cap >= need) return true;
  size_t want = std::max<size_t>(need, 4096);
  if (!s->recorded) {
    if (s->ptr) release(s->ptr);
    *s = tb_scratch{};
    void* p = alloc(want);
    if (!p) return false;
    s->ptr = p;
    s->cap = want;
    return true;
  }
  try {
    kept->reserve(kept->size() + 1);
  } catch (...) {
    return false;
  }
  void* p = nullptr;
  if (2 * s->cap > want && (p = alloc(2 * s->cap))) want = 2 * s->cap;
  if (!p) p = alloc(want);
  if (!p) return false;
  kept->push_back(s->ptr);
  *s = tb_scratch{p, want, false};
  return true;
}
