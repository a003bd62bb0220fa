#include "host_parallel.hpp"

#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <exception>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

namespace hphi {
namespace {

// Up to seven threads beside the caller's, started when first wanted and kept until the process
// ends: starting one for each plan cost more than it did (its stack and its allocator's arena
// are new memory: spin-1 chain of 10 sites, a handle's opening 1.5 -> 2.2 ms with threads per loop).
class Pool {
 public:
  ~Pool() {
    if (getpid() != pid_) {  // a forked copy: the threads are not there to be joined
      new std::vector<std::thread>(std::move(threads_));
      return;
    }
    {
      std::lock_guard<std::mutex> lock(m_);
      stop_ = true;
    }
    wake_.notify_all();
    for (std::thread &t : threads_) t.join();
  }

  bool run(int64_t n, int helpers, const std::function<void(int64_t)> &f) {
    std::unique_lock<std::mutex> alone(busy_, std::try_to_lock);
    if (!alone || getpid() != pid_) return false;
    {
      std::lock_guard<std::mutex> lock(m_);
      try {
        while ((int)threads_.size() < helpers) threads_.emplace_back([this]() { work(); });
      } catch (const std::system_error &) {  // no more threads: those there are do it
      }
      f_ = &f;
      n_ = n;
      next_ = 0;
      error_ = nullptr;
      wanted_ = std::min(helpers, (int)threads_.size());
    }
    wake_.notify_all();
    items();
    std::unique_lock<std::mutex> lock(m_);
    wanted_ = 0;
    done_.wait(lock, [this]() { return working_ == 0; });
    if (error_) std::rethrow_exception(error_);
    return true;
  }

 private:
  void items() {
    try {
      for (int64_t k; (k = next_++) < n_;) (*f_)(k);
    } catch (...) {
      std::lock_guard<std::mutex> lock(m_);
      if (!error_) error_ = std::current_exception();
      next_ = n_;
    }
  }
  void work() {
    std::unique_lock<std::mutex> lock(m_);
    for (;;) {
      wake_.wait(lock, [this]() { return stop_ || wanted_ > 0; });
      if (stop_) return;
      wanted_--;
      working_++;
      lock.unlock();
      items();
      lock.lock();
      if (--working_ == 0) done_.notify_one();
    }
  }

  const pid_t pid_ = getpid();
  std::mutex busy_, m_;
  std::condition_variable wake_, done_;
  std::vector<std::thread> threads_;
  const std::function<void(int64_t)> *f_ = nullptr;
  int64_t n_ = 0;
  std::atomic<int64_t> next_{0};
  std::exception_ptr error_;
  int wanted_ = 0, working_ = 0;  // helpers still to join, helpers at work
  bool stop_ = false;
};

}  // namespace

void host_parallel(int64_t n, double us, const std::function<void(int64_t)> &f) {
  static Pool pool;
  const int cores = std::max(1, (int)std::thread::hardware_concurrency());
  const int helpers = (int)std::min<int64_t>({7, cores - 1, n - 1, (int64_t)(us / 200.0)});
  if (helpers > 0 && pool.run(n, helpers, f)) return;
  for (int64_t k = 0; k < n; k++) f(k);
}

}  // namespace hphi
