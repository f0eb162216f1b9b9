// copy_pool.h -- the process-wide threads that copy between pageable and
// page-locked host memory (transfer.cpp).
#pragma once

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstddef>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>
#ifdef __SSE2__
#include <emmintrin.h>
#endif

namespace cpsz {

inline void cpu_relax() {
#ifdef __SSE2__
  _mm_pause();
#endif
}

// For a few instructions at a time: workers that all look for a piece at once
// would queue up asleep behind a mutex (a host field's banded upload took 5 %
// longer).
class SpinLock {
 public:
  void lock() {
    for (int n = 0; held_.exchange(true, std::memory_order_acquire); n++) {
      if (n < 100) cpu_relax();
      else std::this_thread::yield();
    }
  }
  void unlock() { held_.store(false, std::memory_order_release); }

 private:
  std::atomic<bool> held_{false};
};

// A job is a number of pieces, work(k) copies piece k.  Its owner opens
// pieces in order as their buffers become free (or full) and waits for single
// ones; the workers take open pieces of any job, so a job whose owner waits
// for the device holds up nobody else's.  A worker without an open piece
// sleeps if there is no job; if there is, it looks for a piece for a
// millisecond, yielding its core to whoever wants it, and then sleeps: waking
// it costs a small transfer more than its copies (1024 x 1100 floats
// decompressed to pageable memory .94 ms, 1.0 to 1.5 with workers that sleep
// after 20 us).  An owner that waits for a piece yields, too.
class CopyPool {
 public:
  // Pieces between the first one not waited for and the last one opened.
  static constexpr int kWindow = 64;

  class Job {
   public:
    template <class Work>
    Job(CopyPool& pool, const Work& work)
        : pool_(pool), arg_(&work), call_([](const void* w, int k) { (*(const Work*)w)(k); }) {
      for (auto& d : done_) d.store(0, std::memory_order_relaxed);
      std::lock_guard<SpinLock> lk(pool_.jobs_);
      pool_.link(this);
      pool_.linked_++;
    }
    // Pieces that no worker has taken are dropped, those taken are finished.
    ~Job() {
      {
        std::lock_guard<SpinLock> lk(pool_.jobs_);
        pool_.unlink(this);
        pool_.linked_--;
      }
      spin([&] { return busy_.load(std::memory_order_acquire) == 0; });
    }
    Job(const Job&) = delete;
    Job& operator=(const Job&) = delete;

    // Pieces below `end` may be copied.
    void open(int end) {
      int more;
      {
        std::lock_guard<SpinLock> lk(pool_.jobs_);
        more = end - open_;
        if (more <= 0) return;
        open_ = end;
      }
      pool_.wake(more);
    }
    // Pieces will be opened within the next millisecond: sleeping workers wake
    // up for them now.
    void arm() { pool_.wake(kWindow); }
    // Returns once piece k, which is open, has been copied.
    void wait(int k) {
      spin([&] { return done_[k % kWindow].load(std::memory_order_acquire) == k + 1; });
    }
    // The owner copies an open piece itself; false: none is left to take.
    bool help_once() {
      const int k = take();
      if (k >= 0) run(k);
      return k >= 0;
    }
    void help() {
      while (help_once()) {
      }
    }

   private:
    friend class CopyPool;
    int take() {
      std::lock_guard<SpinLock> lk(pool_.jobs_);
      return claim();
    }
    int claim() {  // under the pool's lock
      if (next_ >= open_) return -1;
      busy_.fetch_add(1, std::memory_order_relaxed);
      return next_++;
    }
    void run(int k) {
      call_(arg_, k);
      done_[k % kWindow].store(k + 1, std::memory_order_release);
      busy_.fetch_sub(1, std::memory_order_release);  // the last touch: the owner may go on from here
    }
    template <class Ready>
    static void spin(const Ready& ready) {
      for (int n = 0; !ready(); n++) {
        if (n < 500) cpu_relax();
        else std::this_thread::yield();
      }
    }
    CopyPool& pool_;
    int next_ = 0, open_ = 0;  // under the pool's lock
    std::atomic<int> busy_{0};
    std::atomic<int> done_[kWindow];
    const void* arg_;
    void (*call_)(const void*, int);
    Job *left_ = nullptr, *right_ = nullptr;
  };

  explicit CopyPool(int workers) {
    try {
      for (int w = 0; w < workers; w++) workers_.emplace_back([this] { loop(); });
    } catch (const std::system_error&) {  // no more threads to be had: those that run, or none, will do
    }
  }
  ~CopyPool() {
    stop_ = true;
    wake(kWindow);
    for (auto& t : workers_) t.join();
  }
  static CopyPool& get() {
    static CopyPool p([] {
      const unsigned hw = std::thread::hardware_concurrency();
      return (int)std::min(8u, hw > 1 ? hw - 1 : 0u);
    }());
    return p;
  }
  bool parallel() const { return !workers_.empty(); }

 private:
  // The jobs form a ring in the order they came; workers look from first_ on,
  // which moves past the job a piece was taken from: jobs take turns.
  void link(Job* j) {
    if (!first_) {
      j->left_ = j->right_ = first_ = j;
      return;
    }
    j->right_ = first_;
    j->left_ = first_->left_;
    j->left_->right_ = first_->left_ = j;
  }
  void unlink(Job* j) {
    if (j->right_ == j) {
      first_ = nullptr;
      return;
    }
    j->left_->right_ = j->right_;
    j->right_->left_ = j->left_;
    if (first_ == j) first_ = j->right_;
  }
  Job* claim(int* k) {
    Job* j = first_;
    if (!j) return nullptr;
    do {
      if ((*k = j->claim()) >= 0) {
        first_ = j->right_;
        return j;
      }
      j = j->right_;
    } while (j != first_);
    return nullptr;
  }
  // A worker counts itself asleep before it looks at the epoch, and the epoch
  // moves before the sleepers are counted: one of the two sees the other.
  void wake(int pieces) {
    epoch_.fetch_add(1);
    if (asleep_.load() == 0) return;
    { std::lock_guard<std::mutex> lk(m_); }
    if (pieces == 1) cv_.notify_one();
    else cv_.notify_all();
  }
  void loop() {
    while (!stop_) {
      const unsigned seen = epoch_.load();  // before the look at the jobs
      int k;
      Job* j;
      {
        std::lock_guard<SpinLock> lk(jobs_);
        j = claim(&k);
      }
      if (j) {
        j->run(k);
        continue;
      }
      const auto until = std::chrono::steady_clock::now() + std::chrono::milliseconds(1);
      for (int n = 1; epoch_.load(std::memory_order_acquire) == seen && linked_.load() > 0; n++) {
        if (n < 500) cpu_relax();
        else std::this_thread::yield();
        if (n % 32 == 0 && std::chrono::steady_clock::now() > until) break;
      }
      if (epoch_.load() != seen) continue;
      std::unique_lock<std::mutex> lk(m_);
      asleep_++;
      cv_.wait(lk, [&] { return epoch_.load() != seen; });
      asleep_--;
    }
  }
  SpinLock jobs_;
  Job* first_ = nullptr;
  std::mutex m_;  // with cv_: sleeping workers
  std::condition_variable cv_;
  std::atomic<int> linked_{0}, asleep_{0};  // jobs, sleeping workers
  std::atomic<bool> stop_{false};
  std::atomic<unsigned> epoch_{0};  // moves when pieces are opened
  std::vector<std::thread> workers_;  // last: they use all of the above
};

}  // namespace cpsz
