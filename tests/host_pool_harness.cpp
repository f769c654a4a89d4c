// Exercises fv2d_gb300/csrc/host_pool.hpp: parallel loops from several threads
// at once (every index visited once, sizes around the piece boundaries, no
// workers at all), and the buffer pool's bound and reuse.  Exit code 0: as
// expected.
#include <atomic>
#include <cstdio>

#include "../fv2d_gb300/csrc/host_pool.hpp"

using namespace fv2d;

static bool loops(HostPool &pool, int rounds) {
  for (int r = 0; r < rounds; ++r)
    for (size_t n : {0, 1, 2, 7, 8, 9, 63, 1000})
      for (size_t grain : {1, 3, 64}) {
        std::vector<std::atomic<int>> seen(n);
        std::atomic<size_t> small{0};
        pool.run(n, grain, [&](size_t b, size_t e) {
          if (e - b < grain && n >= grain) ++small;
          for (size_t k = b; k < e; ++k) ++seen[k];
        });
        for (auto &s : seen)
          if (s != 1) return false;
        if (small) return false;
      }
  return true;
}

int main() {
  {
    HostPool none;
    if (!loops(none, 1)) return 1;
  }
  HostPool pool;
  pool.start(5);
  std::atomic<int> bad{0};
  std::vector<std::thread> callers;
  for (int k = 0; k < 4; ++k) callers.emplace_back([&] { bad += !loops(pool, 50); });
  for (auto &t : callers) t.join();
  if (bad) return 2;

  BufferPool buffers;
  const size_t big = BufferPool::kKeep / sizeof(float) / 2;
  BufferPool::Buffer a = buffers.take(1000), b = buffers.take(big), c = buffers.take(big), d = buffers.take(big);
  if (a.size != 1000 || !b.data || !c.data || !d.data) return 3;
  const float *pa = a.data.get(), *pd = d.data.get();
  buffers.give(std::move(a));
  if (buffers.take(2000).data.get() == pa) return 4;  // too small for it
  a = buffers.take(600);                              // large enough, and not more than twice the size
  if (a.data.get() != pa || a.size != 1000) return 5;
  buffers.give(std::move(b));
  buffers.give(std::move(c));
  buffers.give(std::move(d));  // over the bound: the oldest goes
  if (buffers.take(big).size != big) return 6;
  BufferPool::Buffer e = buffers.take(big);
  if (e.data.get() != pd && !e.data) return 7;
  return 0;
}
