// BufferPool (fv2d_gb300/csrc/host_pool.hpp): what it keeps.  The bytes it holds
// after each call, the buffer a call gets back, and, over the bound, that the
// oldest buffers go and no others.  Prints the step that failed; exit code 0: as
// expected.
#include <cstdio>

#include "../fv2d_gb300/csrc/host_pool.hpp"

using fv2d::BufferPool;

#define CHECK(step, what)      \
  if (!(what)) {               \
    std::printf("%d\n", step); \
    return 1;                  \
  }

int main() {
  constexpr size_t half = BufferPool::kKeep / sizeof(float) / 2;
  BufferPool pool;
  BufferPool::Buffer small = pool.take(1000), b = pool.take(half), c = pool.take(half), d = pool.take(half);
  const float *ps = small.data.get(), *pc = c.data.get(), *pd = d.data.get();
  CHECK(1, ps && b.data && pc && pd && pool.kept() == 0)
  pool.give(std::move(small));
  CHECK(2, pool.kept() == 1000 * sizeof(float))
  pool.give(std::move(b));
  CHECK(3, pool.kept() == half * sizeof(float) + 1000 * sizeof(float))
  pool.give(std::move(c));  // over the bound: the oldest, the small one, goes
  CHECK(4, pool.kept() == 2 * half * sizeof(float))
  pool.give(std::move(d));  // and b
  CHECK(5, pool.kept() == 2 * half * sizeof(float))
  BufferPool::Buffer x = pool.take(half), y = pool.take(half);
  CHECK(6, pool.kept() == 0)
  const float *px = x.data.get(), *py = y.data.get();
  CHECK(7, (px == pc && py == pd) || (px == pd && py == pc))
  pool.give(std::move(x));
  BufferPool::Buffer z = pool.take(half / 2 - 1);  // not one more than twice its size
  CHECK(8, z.size == half / 2 - 1 && pool.kept() == half * sizeof(float))
  z = pool.take(half / 2);
  CHECK(9, z.size == half && z.data.get() == px && pool.kept() == 0)
  BufferPool::Buffer big = pool.take(2 * half + 1);  // larger than all that may be kept
  CHECK(10, big.data)
  pool.give(std::move(big));
  pool.give(BufferPool::Buffer());
  CHECK(11, pool.kept() == 0)
  return 0;
}
