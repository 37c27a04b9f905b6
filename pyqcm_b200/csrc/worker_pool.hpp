// A pool of host threads that live for the whole process (host code).
#pragma once
#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstdint>
#include <deque>
#include <functional>
#include <future>
#include <mutex>
#include <system_error>
#include <thread>

namespace qed {

// Worker threads kept for the life of the process, so that each keeps its
// Workspace (stream, reduction buffers, pinned staging) from one batch call to
// the next. A batch call hands the pool one work loop that `extra` workers and
// the calling thread run; batch calls from different host threads take turns.
// Its threads are detached and wait on its members for the rest of the
// process, so a pool is never destroyed (the library's pools are leaked
// singletons).
class WorkerPool {
 public:
  void run(int extra, const std::function<void()> &work) {
    std::lock_guard<std::mutex> serial(run_mtx_);
    run_locked(extra, work);
  }
  // the same unless another call has the pool: then nothing, and false
  bool try_run(int extra, const std::function<void()> &work) {
    std::unique_lock<std::mutex> serial(run_mtx_, std::try_to_lock);
    if (!serial) return false;
    run_locked(extra, work);
    return true;
  }

 private:
  void run_locked(int extra, const std::function<void()> &work) {
    {
      std::lock_guard<std::mutex> l(m_);
      while ((int)threads_ < extra) {
        const int idx = (int)threads_++;
        std::thread([this, idx] { loop(idx); }).detach();
      }
      job_ = work;
      wanted_ = extra;
      active_ = extra;
      ++gen_;
    }
    cv_.notify_all();
    work();
    std::unique_lock<std::mutex> l(m_);
    done_.wait(l, [&] { return active_ == 0; });
    job_ = nullptr;
  }
  void loop(int idx) {
    uint64_t seen = 0;
    std::unique_lock<std::mutex> l(m_);
    for (;;) {
      cv_.wait(l, [&] { return gen_ != seen; });
      seen = gen_;
      if (idx >= wanted_) continue;
      std::function<void()> w = job_;
      l.unlock();
      w();
      l.lock();
      if (--active_ == 0) done_.notify_all();
    }
  }
  std::mutex run_mtx_, m_;
  std::condition_variable cv_, done_;
  std::function<void()> job_;
  size_t threads_ = 0;
  int wanted_ = 0, active_ = 0;
  uint64_t gen_ = 0;
};

// A queue of independent tasks, taken in order by threads that are started as they are
// needed, up to `most`, and live for the rest of the process (like a WorkerPool, it is
// never destroyed). Without any thread a task runs where it is submitted.
template <class T> class TaskQueue {
 public:
  explicit TaskQueue(int most) : most_(most) {}
  std::future<T> submit(std::function<T()> f) {
    std::packaged_task<T()> t(std::move(f));
    std::future<T> r = t.get_future();
    std::unique_lock<std::mutex> l(m_);
    if (idle_ <= (int)q_.size() && threads_ < most_) {
      try {
        std::thread([this] { loop(); }).detach();
        ++threads_;
      } catch (const std::system_error &) {  // no thread to be had
      }
    }
    if (!threads_) {
      l.unlock();
      t();
      return r;
    }
    q_.push_back(std::move(t));
    cv_.notify_one();
    return r;
  }

 private:
  void loop() {
    std::unique_lock<std::mutex> l(m_);
    for (;;) {
      ++idle_;
      cv_.wait(l, [&] { return !q_.empty(); });
      --idle_;
      std::packaged_task<T()> t = std::move(q_.front());
      q_.pop_front();
      l.unlock();
      t();
      t = std::packaged_task<T()>();  // what it holds goes with it
      l.lock();
    }
  }
  const int most_;
  std::mutex m_;
  std::condition_variable cv_;
  std::deque<std::packaged_task<T()>> q_;
  int threads_ = 0, idle_ = 0;
};

// Runs call(0) .. call(n - 1) on up to `threads` threads of the pool and waits for
// them; false if the pool was taken (then none ran) or a call returned false (then no
// further one is started). After a failed call its thread runs drain() before the
// caller goes on: a call that was left by an exception may have work on its thread's
// stream that reads what the caller frees next.
template <class Call, class Drain>
bool run_parts(WorkerPool &pool, int threads, int n, Call &&call, Drain &&drain) {
  std::atomic<int> next{0};
  std::atomic<bool> ok{true};
  auto work = [&] {
    for (int i = next++; i < n && ok; i = next++)
      if (!call(i)) {
        ok = false;
        drain();
      }
  };
  return pool.try_run(std::max(1, std::min(threads, n)) - 1, work) && ok;
}

}  // namespace qed
