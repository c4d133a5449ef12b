// sr_parallel.hpp — host-side parallel passes: a fork-join helper for one-off
// passes, and a pool of waiting workers for the passes of every call.
#pragma once
#include <algorithm>
#include <condition_variable>
#include <cstdint>
#include <functional>
#include <mutex>
#include <system_error>
#include <thread>
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
// of them took 0.3 ms of every call.  One thread at a time calls run() (a
// context serves one caller at a time).
class WorkerPool {
 public:
  WorkerPool() = default;
  WorkerPool(const WorkerPool &) = delete;
  WorkerPool &operator=(const WorkerPool &) = delete;
  ~WorkerPool() {
    {
      std::lock_guard<std::mutex> lock(m_);
      stop_ = true;
    }
    wake_.notify_all();
    for (auto &t : workers_) t.join();
  }

  // fn(0) .. fn(chunks - 1), each once, on the caller and up to `threads` - 1
  // workers; returns when all are done.
  void run(int chunks, int threads, const std::function<void(int)> &fn) {
    if (chunks <= 1 || threads <= 1) {
      for (int c = 0; c < chunks; ++c) fn(c);
      return;
    }
    grow(std::min(threads, chunks) - 1);
    {
      std::lock_guard<std::mutex> lock(m_);
      fn_ = &fn;
      chunks_ = chunks;
      next_ = 0;
      pending_ = chunks;
      ++generation_;
    }
    wake_.notify_all();
    work(fn);
    std::unique_lock<std::mutex> lock(m_);
    done_.wait(lock, [&] { return pending_ == 0; });
    fn_ = nullptr;
  }

 private:
  void grow(int want) {
    while (static_cast<int>(workers_.size()) < want) {
      try {
        workers_.emplace_back([this] { loop(); });
      } catch (const std::system_error &) {
        return;  // fewer workers; the caller takes the remaining chunks
      }
    }
  }
  // Takes chunks until none is left.
  void work(const std::function<void(int)> &fn) {
    for (;;) {
      int c;
      {
        std::lock_guard<std::mutex> lock(m_);
        if (fn_ != &fn || next_ >= chunks_) return;
        c = next_++;
      }
      fn(c);
      std::lock_guard<std::mutex> lock(m_);
      if (--pending_ == 0) done_.notify_all();
    }
  }
  void loop() {
    uint64_t seen = 0;
    for (;;) {
      const std::function<void(int)> *fn;
      {
        std::unique_lock<std::mutex> lock(m_);
        wake_.wait(lock, [&] { return stop_ || (fn_ && generation_ != seen); });
        if (stop_) return;
        seen = generation_;
        fn = fn_;
      }
      work(*fn);
    }
  }

  std::mutex m_;
  std::condition_variable wake_, done_;
  std::vector<std::thread> workers_;
  const std::function<void(int)> *fn_ = nullptr;
  int chunks_ = 0, next_ = 0, pending_ = 0;
  uint64_t generation_ = 0;
  bool stop_ = false;
};

}  // namespace sr
