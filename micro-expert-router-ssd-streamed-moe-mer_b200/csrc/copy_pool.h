// Host threads that fill the pinned staging buffers of an admission: one thread copies pageable memory at about 11 GB/s, a fifth
// of what the PCIe link takes.  A pool belongs to one backend, is created on its first large pageable admission, holds at
// most MAX_WORKERS threads that sleep between admissions, and ends with the backend.
#pragma once

#include <sched.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <functional>
#include <mutex>
#include <thread>
#include <vector>

class CopyPool {
 public:
  static constexpr unsigned MAX_WORKERS = 8;

  CopyPool() {
    cpu_set_t set;
    CPU_ZERO(&set);
    const int cpus = sched_getaffinity(0, sizeof set, &set) == 0 ? CPU_COUNT(&set) : 1;
    const unsigned n = std::min<unsigned>(MAX_WORKERS, (unsigned)std::max(cpus - 1, 0));  // the caller copies too
    try {
      for (unsigned i = 0; i < n; i++) threads_.emplace_back([this] { loop(); });
    } catch (...) {  // fewer threads are to be had: the caller and those that started do the work
    }
  }
  ~CopyPool() {
    {
      std::lock_guard<std::mutex> l(mu_);
      stop_ = true;
    }
    wake_.notify_all();
    for (auto &t : threads_) t.join();
  }
  CopyPool(const CopyPool &) = delete;
  CopyPool &operator=(const CopyPool &) = delete;

  // Every worker runs `job` once; wait() returns when all of them have left it.
  void start(const std::function<void()> *job) {
    std::lock_guard<std::mutex> l(mu_);
    job_ = job, running_ = threads_.size(), epoch_++;
    wake_.notify_all();
  }
  void wait() {
    std::unique_lock<std::mutex> l(mu_);
    idle_.wait(l, [this] { return running_ == 0; });
    job_ = nullptr;
  }

 private:
  void loop() {
    uint64_t seen = 0;
    std::unique_lock<std::mutex> l(mu_);
    for (;;) {
      wake_.wait(l, [&] { return stop_ || epoch_ != seen; });
      if (stop_) return;
      seen = epoch_;
      const std::function<void()> *job = job_;
      l.unlock();
      (*job)();
      l.lock();
      if (--running_ == 0) idle_.notify_all();
    }
  }

  std::vector<std::thread> threads_;
  std::mutex mu_;
  std::condition_variable wake_, idle_;
  const std::function<void()> *job_ = nullptr;
  size_t running_ = 0;
  uint64_t epoch_ = 0;
  bool stop_ = false;
};
