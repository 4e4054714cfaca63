// listpolicy.cuh - how a context's steps go on after a step that could not be
// finished on its neighbour lists (pairlist.cuh).  Host code without CUDA.
#pragma once

#include <algorithm>
#include <cstdint>

namespace tg {

// Why a step could not be finished on its neighbour lists.
constexpr uint32_t kStopMoved = 1u;     // a particle moved beyond the bound
constexpr uint32_t kStopCapacity = 2u;  // a list outgrew its capacity

// The stopped step, or chain of steps, is taken on the cell walk (a sort and a
// walk per stage), and the next ones on lists again, with more of what was
// short.  Stops that
// come close together lengthen the walk, so that a state for which lists do
// not work at all pays for one attempt in kLongest steps; steps without a
// stop bring back the narrow margin and the chains.
struct ListPolicy {
  static constexpr float kMargin = 0.005f, kWidest = 0.08f;  // in support radii
  static constexpr int kLongest = 256;                       // steps on the walk
  static constexpr int kBatch = 256, kFirstBatch = 8;
  static constexpr int64_t kPatience = 64, kMostPatience = 4096;

  float margin = kMargin;  // the accelerations' share of the displacement bound
  double room = 1.0;       // of the lists' capacity
  bool chains = true;      // steps may share their lists
  int walk = 0;            // steps to take on the cell walk next
  int length = 0;          // of the last walk
  // Steps enqueued before the host looks for a stop: what a stop wastes, as
  // the steps behind it do nothing.
  int batch = kBatch;
  int64_t since = 0;             // steps on lists since the last stop
  int64_t clean = 0;             // ... or the last easing
  int64_t patience = kPatience;  // of them before the margin or chains ease
  bool eased = false;

  // steps: those that were to share the lists.
  void stopped(uint32_t why, int steps) {
    if ((why & kStopMoved) != 0u) {
      margin = std::min(2.f * margin, kWidest);
      chains = false;
    }
    if ((why & kStopCapacity) != 0u) room *= 1.5;
    length = length > 0 && since < 16 * length ? std::min(2 * length, kLongest)
                                              : steps;
    walk = length;
    if (eased && clean < patience) patience = std::min(2 * patience, kMostPatience);
    eased = false;
    since = clean = 0;
    batch = kFirstBatch;
  }
  void walked(int steps) { walk -= steps; }
  // True when the margin or the chains changed.
  bool finished(int steps) {
    since += steps;
    clean += steps;
    batch = std::min(2 * batch, kBatch);
    if (clean < patience || (margin <= kMargin && chains)) return false;
    if (!chains) {
      chains = true;
    } else {
      margin = std::max(0.5f * margin, kMargin);
    }
    eased = true;
    clean = 0;
    return true;
  }
};

}  // namespace tg
