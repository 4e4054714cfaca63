// The buffers of the list steps are held all together or not at all, whichever
// allocation fails and however often they are asked for.
#include <cstdio>
#include <cstdlib>
#include <map>

#include "listbuf.cuh"

namespace {

std::map<void*, size_t> live;
int countdown = -1;  // allocations until one fails; -1: none does

void* alloc(size_t bytes) {
  if (countdown == 0) return nullptr;
  if (countdown > 0) --countdown;
  void* p = std::malloc(bytes);
  live[p] = bytes;
  return p;
}
void release(void* p) {
  if (live.erase(p) != 1) std::abort();
  std::free(p);
}

bool complete(const tg::ListBuffers& L, const size_t (&bytes)[tg::kListBufs]) {
  for (int b = 0; b < tg::kListBufs; ++b) {
    if ((L.p[b] != nullptr) != (bytes[b] != 0)) return false;
    if (L.p[b] != nullptr && live[L.p[b]] != bytes[b]) return false;
  }
  return true;
}

#define CHECK(x)                                              \
  do {                                                        \
    if (!(x)) {                                               \
      std::fprintf(stderr, "line %d: %s\n", __LINE__, #x);    \
      return 1;                                               \
    }                                                         \
  } while (0)

}  // namespace

int main() {
  for (const size_t pos : {size_t{0}, size_t{32}}) {  // compensated form, plain form
    const size_t bytes[tg::kListBufs] = {64, 8, 48, pos, 16};
    const int wanted = pos != 0 ? 5 : 4;
    for (int fail = 0; fail < wanted; ++fail) {
      tg::ListBuffers L;
      countdown = fail;
      CHECK(!L.take(bytes, alloc, release));
      CHECK(!L.held() && live.empty());
      for (const void* p : L.p) CHECK(p == nullptr);
      // The next attempt holds every buffer.
      countdown = -1;
      CHECK(L.take(bytes, alloc, release));
      CHECK(L.held() && complete(L, bytes));
      // So does one for longer lists, and a failed one keeps nothing.
      size_t more[tg::kListBufs];
      for (int b = 0; b < tg::kListBufs; ++b) more[b] = bytes[b];
      more[tg::kListEntries] *= 2;
      CHECK(L.take(more, alloc, release) && complete(L, more));
      CHECK(static_cast<int>(live.size()) == wanted);
      countdown = fail;
      CHECK(!L.take(bytes, alloc, release) && !L.held() && live.empty());
      countdown = -1;
    }
  }
  std::puts("ok");
  return 0;
}
