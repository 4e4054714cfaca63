// listbuf.cuh - the device buffers of steps on neighbour lists (pairlist.cuh).
// Host code without CUDA, so that a failing allocation can be tested anywhere.
#pragma once

#include <cstddef>

namespace tg {

// The list entries and their counts, the second data and position records,
// and the paths within a chain.
enum ListBuf { kListEntries = 0, kListCounts, kListDat, kListPos, kListTravel, kListBufs };

// All the buffers that a step needs, or none.
struct ListBuffers {
  void* p[kListBufs] = {};

  bool held() const { return p[kListEntries] != nullptr; }

  // Takes a buffer of every size that is not 0 from alloc(bytes), null when
  // there is none; then those taken go back to release and none is held.
  template<class Alloc, class Release>
  bool take(const size_t (&bytes)[kListBufs], Alloc&& alloc, Release&& release) {
    drop(release);
    for (int b = 0; b < kListBufs; ++b) {
      if (bytes[b] == 0) continue;
      p[b] = alloc(bytes[b]);
      if (p[b] == nullptr) {
        drop(release);
        return false;
      }
    }
    return held();
  }
  template<class Release>
  void drop(Release&& release) {
    for (void*& q : p) {
      if (q != nullptr) release(q);
      q = nullptr;
    }
  }
};

}  // namespace tg
