// BufPool against a fake device of 100 units: reuse, eviction in order of age, release on a failed
// allocation. Prints "pool ok".
#include <cstdio>
#include <cstdlib>
#include <set>

#include "../../dumato_b200/csrc/buf_pool.hpp"

static size_t used = 0;
static std::map<void*, size_t> live;
static int failures = 0;

#define CHECK(x)                                              \
  do {                                                        \
    if (!(x)) {                                               \
      std::printf("line %d: %s\n", __LINE__, #x);             \
      ++failures;                                             \
    }                                                         \
  } while (0)

int main() {
  dmb::BufPool pool(
      40,
      [](void** p, size_t n) {
        if (used + n > 100) return 2;
        *p = std::malloc(1);
        live[*p] = n;
        used += n;
        return 0;
      },
      [](void* p) {
        used -= live.at(p);
        live.erase(p);
        std::free(p);
      });
  void *a = nullptr, *b = nullptr, *c = nullptr, *d = nullptr;
  CHECK(pool.take(&a, 20) == 0 && pool.take(&b, 15) == 0 && used == 35);
  CHECK(pool.give(a) && pool.give(b) && pool.pooled() == 35 && used == 35);
  // best fit, at most twice the size asked for
  CHECK(pool.take(&c, 14) == 0 && c == b && pool.pooled() == 20 && used == 35);
  CHECK(pool.take(&d, 9) == 0 && d != a && used == 44);  // 20 is more than twice 9
  // a buffer beyond the limit goes back to the device, one within it takes the place of the oldest
  void* big = nullptr;
  CHECK(pool.take(&big, 50) == 0 && used == 94);
  CHECK(pool.give(big) && used == 44 && pool.pooled() == 20);
  CHECK(pool.give(c) && pool.pooled() == 35);                 // 20 (a), 15 (c)
  CHECK(pool.give(d) && pool.pooled() == 24 && used == 24);   // a, the oldest, went: 15 + 9
  CHECK(live.count(a) == 0);
  // no room on the device: what is kept is released and the allocation tried again
  void* most = nullptr;
  CHECK(pool.take(&most, 90) == 0 && used == 90 && pool.pooled() == 0);
  void* more = nullptr;
  CHECK(pool.take(&more, 20) == 2 && used == 90);             // nothing to release: the error comes back
  CHECK(pool.give(most) && used == 0);
  int other = 0;
  CHECK(!pool.give(&other));
  // random use never exceeds either limit, never hands a buffer out twice
  std::set<void*> out;
  for (int i = 0; i < 20000; ++i) {
    if (std::rand() % 2 || out.empty()) {
      void* p = nullptr;
      const size_t n = 1 + std::rand() % 12;
      if (pool.take(&p, n) == 0) {
        CHECK(out.insert(p).second && live.at(p) >= n);
      }
    } else {
      void* p = *out.begin();
      out.erase(out.begin());
      CHECK(pool.give(p));
    }
    CHECK(pool.pooled() <= 40 && used <= 100);
  }
  for (void* p : out) pool.give(p);
  CHECK(pool.drop() <= 40 && used == 0 && pool.drop() == 0);
  if (!failures) std::printf("pool ok\n");
  return failures != 0;
}
