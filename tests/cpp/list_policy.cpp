// How many steps walk cells after a stop, and what comes back when: one stop
// costs its chain, frequent ones are tried ever more rarely, and neither the
// margin nor the chains stay changed.
#include <cstdint>
#include <cstdio>

#include "listpolicy.cuh"

namespace {

#define CHECK(x)                                              \
  do {                                                        \
    if (!(x)) {                                               \
      std::fprintf(stderr, "line %d: %s\n", __LINE__, #x);    \
      return 1;                                               \
    }                                                         \
  } while (0)

struct Run {
  int64_t walked = 0, on_lists = 0, idle = 0, stops = 0;
  int widest = 0;
};

// `steps` steps of one call; stop(step, P) says whether a step on lists stops.
template<class Stop>
Run run(tg::ListPolicy& P, int64_t steps, Stop&& stop) {
  Run r;
  int64_t at = 0;
  while (at < steps) {
    const int64_t left = steps - at;
    if (P.walk > 0) {
      const int n = static_cast<int>(left < P.walk ? left : P.walk);
      at += n;
      r.walked += n;
      P.walked(n);
      continue;
    }
    const int n = static_cast<int>(left < P.batch ? left : P.batch);
    int done = 0;
    uint32_t why = 0;
    while (done < n && (why = stop(at + done, P)) == 0u) ++done;
    at += done;
    r.on_lists += done;
    if (why != 0u) {
      ++r.stops;
      r.idle += n - done;  // enqueued, and left the state alone
      P.stopped(why, P.chains && left - done > 1 ? 2 : 1);
    } else {
      P.finished(n);
    }
  }
  return r;
}

}  // namespace

int main() {
  const float base = tg::ListPolicy{}.margin;
  {  // One stop in the third of 1000 steps, and the same in a chain of calls.
    tg::ListPolicy P;
    const Run r = run(P, 1000, [](int64_t s, const tg::ListPolicy& Q) {
      return s == 2 && Q.margin <= 0.005f ? tg::kStopMoved : 0u;
    });
    CHECK(r.stops == 1 && r.walked == 2 && r.on_lists == 998);
    CHECK(r.idle <= tg::ListPolicy::kBatch);
    CHECK(P.chains && P.margin == base && P.walk == 0);
  }
  {  // A capacity stop leaves the margin and the chains alone.
    tg::ListPolicy P;
    P.stopped(tg::kStopCapacity, 1);
    CHECK(P.room == 1.5 && P.margin == base && P.chains && P.walk == 1);
  }
  {  // Lists that never work: one attempt in many steps, and a bounded margin.
    tg::ListPolicy P;
    const Run r = run(P, 100000, [](int64_t, const tg::ListPolicy&) { return tg::kStopMoved; });
    CHECK(r.walked == 100000);
    CHECK(r.stops <= 100000 / tg::ListPolicy::kLongest + 12);
    CHECK(P.margin <= tg::ListPolicy::kWidest);
    // Afterwards they come back, within a call or a driver's one-step calls.
    int64_t slow = 0;
    for (int64_t s = 0; s < 2000; ++s) {
      slow += run(P, 1, [](int64_t, const tg::ListPolicy&) { return 0u; }).walked;
    }
    CHECK(slow <= tg::ListPolicy::kLongest);
    CHECK(P.chains && P.margin == base);
  }
  {  // A state that needs four times the margin for good: few steps repeated.
    tg::ListPolicy P;
    const Run r = run(P, 100000, [](int64_t, const tg::ListPolicy& Q) {
      return Q.margin < 0.02f ? tg::kStopMoved : 0u;
    });
    CHECK(r.walked + r.stops < 500);
  }
  {  // Stops far apart cost a chain each.
    tg::ListPolicy P;
    const Run r = run(P, 10000, [](int64_t s, const tg::ListPolicy& Q) {
      return s % 500 == 499 && Q.walk == 0 ? tg::kStopCapacity : 0u;
    });
    CHECK(r.walked <= 2 * r.stops && r.stops <= 20);
  }
  std::puts("ok");
  return 0;
}
