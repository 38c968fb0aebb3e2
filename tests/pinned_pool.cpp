// The pool of pinned blocks (pinned.cuh) on a counting allocator; every check
// that fails names itself.
#include "pinned.cuh"

#include <cstdio>
#include <cstdlib>
#include <thread>

using namespace picard;

static std::mutex g_mu;
static size_t g_live = 0, g_limit = ~size_t(0);
struct Counting {
  static void* alloc(size_t bytes) {
    std::lock_guard<std::mutex> lk(g_mu);
    if (g_live + bytes > g_limit) return nullptr;
    size_t* p = static_cast<size_t*>(std::malloc(16));
    *p = bytes;
    g_live += bytes;
    return p;
  }
  static void free(void* p) {
    std::lock_guard<std::mutex> lk(g_mu);
    g_live -= *static_cast<size_t*>(p);
    std::free(p);
  }
};
using Pool = PinnedPool<Counting>;

static int bad = 0;
#define CHECK(what, cond) \
  if (!(cond)) std::printf("failed: %s (%zu bytes live)\n", what, g_live), bad = 1

static void fill(Pool& P, int cls, int n) {
  std::vector<void*> b;
  for (int i = 0; i < n; ++i) b.push_back(P.get(cls));
  for (void* p : b) P.put(cls, p);
}

int main() {
  const size_t big = kPinnedBlock[1];
  Pool P;
  fill(P, 1, 3);
  CHECK("nothing kept without a context or an allowance", g_live == 0);
  P.context(1);
  fill(P, 1, 9);
  CHECK("four blocks while a context lives", g_live == 4 * big);
  fill(P, 1, 4);
  CHECK("kept blocks serve the next calls", g_live == 4 * big);
  P.context(-1);
  CHECK("none after the last context", g_live == 0);
  P.set_keep(0, 3 * big);
  fill(P, 1, 9);
  CHECK("the allowance of a device", g_live == 3 * big);
  P.set_keep(1, big);
  CHECK("another device's smaller value takes nothing away", g_live == 3 * big);
  P.set_keep(0, 0);
  CHECK("its own does", g_live == big);
  P.set_keep(1, 0);
  CHECK("no allowance left", g_live == 0);
  P.set_keep(3, ~size_t(0));
  fill(P, 1, 40);
  CHECK("never more than the bound", g_live == kPinnedKeepMost);
  P.set_keep(3, 0);
  g_limit = 2 * big;
  void* a = P.get(1);
  void* b = P.get(1);
  CHECK("an allocation that fails is null", a && b && !P.get(1));
  P.put(1, a);
  P.put(1, b);
  P.put(0, nullptr);
  g_limit = ~size_t(0);
  P.context(1);
  std::vector<std::thread> ts;
  for (int t = 0; t < 4; ++t)
    ts.emplace_back([&P, t] {
      for (int i = 0; i < 500; ++i) fill(P, (t + i) & 1, 3);
    });
  for (auto& t : ts) t.join();
  CHECK("bounded with several threads", g_live <= 4 * big);
  P.context(-1);
  CHECK("all given back", g_live == 0);
  return bad;
}
