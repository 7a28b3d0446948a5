// Host check of the batched path's pools of CUDA streams and events (csrc/handle_pool.hpp): an object
// is handed out on the device it was made on and on no other, also from several threads.
#include <cstdio>
#include <thread>
#include <vector>

#include "handle_pool.hpp"

static int failures = 0;
#define EXPECT(c) \
  do { \
    if (!(c)) { \
      ++failures; \
      std::printf("line %d: %s\n", __LINE__, #c); \
    } \
  } while (0)

struct Obj {
  int device;
};

int main() {
  sov::HandlePool<Obj*> pool;
  int made = 0;
  auto take = [&](int dev) {
    return pool.take(dev, [&] {
      ++made;
      return new Obj{dev};
    });
  };
  // one solve on device 0, then on device 1, then on both again
  Obj* a = take(0);
  pool.give(a);
  Obj* b = take(1);
  EXPECT(b != a && b->device == 1 && made == 2);
  pool.give(b);
  EXPECT(take(0) == a && take(1) == b && made == 2);
  // given back in the other order than taken: each to its own list
  Obj* c = take(1);
  Obj* d = take(0);
  EXPECT(c->device == 1 && d->device == 0 && made == 4);
  for (Obj* o : {d, b, c, a}) pool.give(o);
  for (int k = 0; k < 2; ++k) EXPECT(take(1)->device == 1 && take(0)->device == 0);
  EXPECT(made == 4);
  // threads on three devices
  sov::HandlePool<Obj*> shared;
  std::vector<int> wrong(6, 0);
  std::vector<std::thread> ts;
  for (int t = 0; t < 6; ++t)
    ts.emplace_back([&, t] {
      for (int k = 0; k < 2000; ++k) {
        Obj* o = shared.take(t % 3, [&] { return new Obj{t % 3}; });
        wrong[t] += o->device != t % 3;
        shared.give(o);
      }
    });
  for (std::thread& t : ts) t.join();
  for (int w : wrong) EXPECT(w == 0);
  std::printf("failures %d\n", failures);
  return failures != 0;
}
