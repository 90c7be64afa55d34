// A context's scratch memory: one block that grows on demand.  A recorded launch sequence holds the block's address for as long as
// it may be replayed, so a block that a recording used is not given back when a later call outgrows it; it is kept until the context
// closes (the owner of a shared stream can record too, so the end of a recording is not always seen).  A block that no recording used
// is released at once.  Where a block is kept, the next one is half as large again at least, so that all kept blocks together are at
// most twice the size of the one in use, however often a program records and grows.
#pragma once
#include <stdint.h>

#include <vector>

namespace p0p {

struct Scratch {
  void* ptr = nullptr;
  uint64_t bytes = 0;
  bool recorded = false;            // a recording holds `ptr`
  std::vector<void*> kept;
  // `need` > bytes.  alloc(void**, size) returns 0 or an error, release(void*) frees.  On an error a kept block stays the one in use.
  template <class Alloc, class Release>
  int grow(uint64_t need, Alloc alloc, Release release) {
    const uint64_t mb = 1ull << 20, want = need < 8u * mb ? 8u * mb : (need + mb - 1u) & ~(mb - 1u);
    void* p = nullptr;
    if (!recorded) {
      if (ptr) release(ptr);
      ptr = nullptr; bytes = 0;
      const int e = alloc(&p, want);
      if (e) return e;
      ptr = p; bytes = want;
      return 0;
    }
    uint64_t size = want < bytes + bytes / 2u ? bytes + bytes / 2u : want;
    int e = alloc(&p, size);
    if (e && size > want) e = alloc(&p, size = want);
    if (e) return e;
    kept.push_back(ptr);
    ptr = p; bytes = size; recorded = false;
    return 0;
  }
  template <class Release>
  void clear(Release release) {
    if (ptr) release(ptr);
    for (void* p : kept) release(p);
    ptr = nullptr; bytes = 0; kept.clear();
  }
};

}  // namespace p0p
