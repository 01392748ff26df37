// Host threads that fill the pinned staging memory of an admission: one thread copies pageable memory at about 11 GB/s, a fifth
// of what the PCIe link takes.  A pool belongs to one backend, is created on its first large pageable admission, holds at
// most MAX_WORKERS threads, and ends with the backend.  Waking a sleeping thread costs 50 to 100 us in a virtual machine,
// about what a 5 MB expert takes on the link: after a job the workers stay awake for SPIN_US, so that a run of admissions
// finds them running, and nobody ever waits for a worker that woke too late to find work (jobs are shared, not borrowed).
#pragma once

#include <sched.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <functional>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

class CopyPool {
 public:
  static constexpr unsigned MAX_WORKERS = 6;
  static constexpr int SPIN_US = 500;
  using Job = std::shared_ptr<const std::function<void()>>;  // owns everything it touches once its work is done

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
      epoch_.fetch_add(1);
    }
    wake_.notify_all();
    for (auto &t : threads_) t.join();
  }
  CopyPool(const CopyPool &) = delete;
  CopyPool &operator=(const CopyPool &) = delete;

  // Every worker that is awake, or wakes in time, runs `job` once.
  void start(Job job) {
    bool sleepers;
    {
      std::lock_guard<std::mutex> l(mu_);
      job_ = std::move(job);
      epoch_.fetch_add(1, std::memory_order_release);
      sleepers = sleeping_ > 0;
    }
    if (sleepers) wake_.notify_all();
  }
  // Lets go of the current job.
  void finish() {
    std::lock_guard<std::mutex> l(mu_);
    job_.reset();
  }

 private:
  void loop() {
    uint64_t seen = 0;
    for (;;) {
      const auto until = std::chrono::steady_clock::now() + std::chrono::microseconds(SPIN_US);
      while (epoch_.load(std::memory_order_acquire) == seen && std::chrono::steady_clock::now() < until) std::this_thread::yield();
      Job job;
      {
        std::unique_lock<std::mutex> l(mu_);
        if (epoch_.load() == seen) {
          sleeping_++;
          wake_.wait(l, [&] { return epoch_.load() != seen; });
          sleeping_--;
        }
        if (stop_) return;
        seen = epoch_.load();
        job = job_;
      }
      if (job) (*job)();
    }
  }

  std::vector<std::thread> threads_;
  std::mutex mu_;
  std::condition_variable wake_;
  Job job_;
  std::atomic<uint64_t> epoch_{0};
  unsigned sleeping_ = 0;
  bool stop_ = false;
};
