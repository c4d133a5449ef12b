// sr_parallel.hpp — host-side parallel passes: a fork-join helper for one-off
// passes, and a pool of waiting workers for the passes of every call.
#pragma once
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstdint>
#include <exception>
#include <functional>
#include <memory>
#include <mutex>
#include <system_error>
#include <thread>
#include <utility>
#include <vector>

namespace sr {

template <class F>
void parallel_for(int64_t n, int threads, F &&fn) {
  if (n <= 0) return;
  const int64_t t = std::max<int64_t>(1, std::min<int64_t>(threads, n));
  if (t == 1) {
    fn(int64_t{0}, n);
    return;
  }
  std::vector<std::thread> pool;
  pool.reserve(static_cast<size_t>(t - 1));
  for (int64_t k = 1; k < t; ++k)
    pool.emplace_back([&, k] { fn(n * k / t, n * (k + 1) / t); });
  fn(int64_t{0}, n / t);
  for (auto &th : pool) th.join();
}

// Workers owned by one context, started when a pass first needs them and
// joined with the context.  Starting a thread costs about 20 us, so forking 15
// of them took 0.3 ms of every call; waking one costs tens of microseconds, so
// a worker that has finished looks out for the next pass of the call for a
// moment before it sleeps.  One thread at a time calls run() (a context serves
// one caller at a time).
class WorkerPool {
 public:
  WorkerPool() = default;
  WorkerPool(const WorkerPool &) = delete;
  WorkerPool &operator=(const WorkerPool &) = delete;
  ~WorkerPool() {
    if (!workers_.empty() && getpid() != owner_) {
      // A forked process holds a copy without the threads: joining them, or
      // destroying what they sleep on, would wait for ever.
      new std::vector<std::thread>(std::move(workers_));
      wake_.release();
      return;
    }
    {
      std::lock_guard<std::mutex> lock(m_);
      stop_ = true;
      generation_.fetch_add(1);
    }
    wake_->notify_all();
    for (auto &t : workers_) t.join();
  }

  // fn(0) .. fn(chunks - 1), each once, on the caller and up to `threads` - 1
  // workers; returns when all are done.  An exception of fn leaves the pool
  // usable and reaches the caller once no worker is inside the pass any more
  // (the first one, when several chunks throw).
  void run(int chunks, int threads, const std::function<void(int)> &fn) {
    if (chunks <= 1 || threads <= 1) {
      for (int c = 0; c < chunks; ++c) fn(c);
      return;
    }
    grow(std::min(threads, chunks) - 1);
    fn_ = &fn;
    chunks_ = chunks;
    next_.store(0);
    pending_.store(chunks);
    failure_ = nullptr;
    failed_.store(false);
    open_.store(true);
    {
      std::lock_guard<std::mutex> lock(m_);
      generation_.fetch_add(1);
    }
    if (sleepers_.load() > 0) wake_->notify_all();
    work();
    // Every chunk done, then no worker left inside the pass: the next one may
    // change its description.
    for (int spin = 0; pending_.load() > 0; ++spin) pause(spin);
    open_.store(false);
    for (int spin = 0; inside_.load() > 0; ++spin) pause(spin);
    if (failure_) std::rethrow_exception(std::exchange(failure_, nullptr));
  }

 private:
  static constexpr int kSpins = 4000;  // about 50 us

  static void pause(int spin) {
    if (spin < kSpins)
      __builtin_ia32_pause();
    else
      std::this_thread::yield();
  }
  void grow(int want) {
    if (workers_.empty()) owner_ = getpid();
    while (static_cast<int>(workers_.size()) < want) {
      try {
        workers_.emplace_back([this] { loop(); });
      } catch (const std::system_error &) {
        return;  // fewer workers; the caller takes the remaining chunks
      }
    }
  }
  void work() {
    for (int c; (c = next_.fetch_add(1)) < chunks_;) {
      try {
        (*fn_)(c);
      } catch (...) {
        if (!failed_.exchange(true)) failure_ = std::current_exception();
      }
      pending_.fetch_sub(1);
    }
  }
  void loop() {
    uint64_t seen = 0;
    for (;;) {
      for (int spin = 0; generation_.load() == seen && spin < kSpins; ++spin) pause(spin);
      if (generation_.load() == seen) {
        std::unique_lock<std::mutex> lock(m_);
        sleepers_.fetch_add(1);
        wake_->wait(lock, [&] { return generation_.load() != seen; });
        sleepers_.fetch_sub(1);
      }
      seen = generation_.load();
      if (stop_.load()) return;
      // The pass's description is read only between entering and leaving, and
      // only while it is open (run() closes it, then waits for both).
      inside_.fetch_add(1);
      if (open_.load()) work();
      inside_.fetch_sub(1);
    }
  }

  std::mutex m_;
  std::unique_ptr<std::condition_variable> wake_{new std::condition_variable};
  std::vector<std::thread> workers_;
  pid_t owner_ = 0;  // the process that started them
  const std::function<void(int)> *fn_ = nullptr;
  int chunks_ = 0;
  std::atomic<int> next_{0}, pending_{0}, inside_{0}, sleepers_{0};
  std::atomic<bool> open_{false}, stop_{false}, failed_{false};
  std::exception_ptr failure_;  // of the pass: written by the one that set failed_
  std::atomic<uint64_t> generation_{0};
};

}  // namespace sr
