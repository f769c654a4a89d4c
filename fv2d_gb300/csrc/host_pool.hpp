// host_pool.hpp -- host-side helpers of the service: a few threads that share
// its bulk copies and conversions, and the memory of finished results, kept
// for the next ones.
#pragma once

#include <algorithm>
#include <condition_variable>
#include <cstddef>
#include <memory>
#include <mutex>
#include <new>
#include <system_error>
#include <thread>
#include <vector>

namespace fv2d {

// Threads that wait for pieces of parallel loops.  Any thread may call run();
// calls from several threads share the workers.
class HostPool {
 public:
  // Starts up to `threads` workers; with fewer (or none) to be had, run()
  // does the rest on the caller.
  void start(int threads) {
    try {
      for (int k = 0; k < threads; ++k) workers_.emplace_back([this] { work(); });
    } catch (const std::system_error &) {
    } catch (const std::bad_alloc &) {
    }
  }
  ~HostPool() {
    {
      std::lock_guard<std::mutex> lock(mu_);
      stop_ = true;
    }
    cv_.notify_all();
    for (std::thread &t : workers_) t.join();
  }

  // fn(begin, end) over [0, n), in pieces of at least `grain`, on the workers
  // and the caller; returns when all of it is done.  fn must not throw.
  template <class F>
  void run(size_t n, size_t grain, const F &fn) {
    const size_t parts = std::max<size_t>(1, std::min(workers_.size() + 1, n / std::max<size_t>(grain, 1)));
    Loop loop;
    loop.fn = [](const void *f, size_t b, size_t e) { (*static_cast<const F *>(f))(b, e); };
    loop.arg = &fn;
    loop.n = n;
    loop.parts = parts;
    if (parts > 1) {
      bool queued = false;
      {
        std::lock_guard<std::mutex> lock(mu_);
        try {
          loops_.push_back(&loop);
          queued = true;
        } catch (const std::bad_alloc &) {
        }
      }
      if (queued) cv_.notify_all();
    }
    std::unique_lock<std::mutex> lock(mu_);
    while (loop.next < parts) step(loop, lock);
    loops_.erase(std::remove(loops_.begin(), loops_.end(), &loop), loops_.end());
    loop.idle.wait(lock, [&] { return loop.done == parts; });
  }

 private:
  struct Loop {
    void (*fn)(const void *, size_t, size_t);
    const void *arg;
    size_t n, parts;
    size_t next = 0, done = 0;  // pieces handed out, pieces finished (under mu_)
    std::condition_variable idle;
  };
  // Runs the loop's next piece; `lock` holds mu_ before and after.
  void step(Loop &l, std::unique_lock<std::mutex> &lock) {
    const size_t p = l.next++;
    lock.unlock();
    l.fn(l.arg, l.n * p / l.parts, l.n * (p + 1) / l.parts);
    lock.lock();
    if (++l.done == l.parts) l.idle.notify_all();
  }
  void work() {
    std::unique_lock<std::mutex> lock(mu_);
    for (;;) {
      Loop *l = nullptr;
      for (Loop *x : loops_)
        if (x->next < x->parts) {
          l = x;
          break;
        }
      if (l)
        step(*l, lock);
      else if (stop_)
        return;
      else
        cv_.wait(lock);
    }
  }
  std::mutex mu_;
  std::condition_variable cv_;
  std::vector<Loop *> loops_;
  std::vector<std::thread> workers_;
  bool stop_ = false;
};

// Result buffers that were given back, up to kKeep bytes: memory fresh from
// the system costs a page fault per page on its first write.  Thread-safe.
class BufferPool {
 public:
  struct Buffer {
    std::unique_ptr<float[]> data;
    size_t size = 0;  // floats
  };
  static constexpr size_t kKeep = (size_t)512 << 20;

  // A buffer of at least n floats (empty when memory runs out).
  Buffer take(size_t n) {
    {
      std::lock_guard<std::mutex> lock(mu_);
      size_t best = free_.size();
      for (size_t k = 0; k < free_.size(); ++k)
        if (free_[k].size >= n && free_[k].size <= 2 * n && (best == free_.size() || free_[k].size < free_[best].size))
          best = k;
      if (best < free_.size()) {
        Buffer b = std::move(free_[best]);
        free_[best] = std::move(free_.back());
        free_.pop_back();
        held_ -= b.size * sizeof(float);
        return b;
      }
    }
    Buffer b;
    b.data.reset(new (std::nothrow) float[n]);
    b.size = b.data ? n : 0;
    return b;
  }
  // Keeps b for a later take(), or frees it: the oldest kept buffers make
  // room for it.
  void give(Buffer b) {
    const size_t bytes = b.size * sizeof(float);
    if (!b.data || bytes > kKeep) return;
    std::vector<Buffer> drop;  // freed after the lock
    std::lock_guard<std::mutex> lock(mu_);
    try {
      while (held_ + bytes > kKeep && !free_.empty()) {
        drop.reserve(drop.size() + 1);
        held_ -= free_.front().size * sizeof(float);
        drop.push_back(std::move(free_.front()));
        free_.erase(free_.begin());
      }
      free_.reserve(free_.size() + 1);
    } catch (const std::bad_alloc &) {
      return;
    }
    held_ += bytes;
    free_.push_back(std::move(b));
  }
  size_t kept() {  // bytes
    std::lock_guard<std::mutex> lock(mu_);
    return held_;
  }

 private:
  std::mutex mu_;
  std::vector<Buffer> free_;
  size_t held_ = 0;
};

}  // namespace fv2d
