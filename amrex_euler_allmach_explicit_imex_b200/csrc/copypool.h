// Host threads that copy rows between a caller's box and pinned memory
// (hoststage.cu).
#pragma once

#include <atomic>
#include <condition_variable>
#include <functional>
#include <mutex>
#include <thread>
#include <vector>

// A fixed set of host threads that run the n tasks of one job together with
// the calling thread; run() returns when every task is done and no thread
// holds the job any more (the job lives on run()'s stack).  A thread that
// cannot be made is done without, down to the calling thread alone.
class CopyPool {
 public:
  explicit CopyPool(int workers)
  {
    try {
      threads_.reserve(workers);
      for (int w = 0; w < workers; ++w) threads_.emplace_back([this] { loop(); });
    } catch (...) {
    }
  }
  ~CopyPool()
  {
    {
      std::lock_guard<std::mutex> lock(mu_);
      stop_ = true;
    }
    cv_.notify_all();
    for (auto& t : threads_) t.join();
  }
  struct Job {
    const std::function<void(int)>* f = nullptr;
    int n = 0;
    std::atomic<int> next{0};
    int helped = 0;  // tasks the caller ran between begin and finish
    int done = 0;   // tasks finished (under mu_)
    int users = 0;  // worker threads holding the job (under mu_)
  };
  void run(int n, const std::function<void(int)>& f)
  {
    Job job;
    job.f = &f;
    job.n = n;
    begin(job);
    finish(job);
  }
  // The two halves of run(): the threads start on the job, the caller joins them
  // on what is left and returns with the last task.
  void begin(Job& job)
  {
    {
      std::lock_guard<std::mutex> lock(mu_);
      job_ = &job;
      ++gen_;
    }
    cv_.notify_all();
  }
  // Between the two, the caller's hand with one task below `limit`; false when
  // there is none left to take.
  bool help(Job& job, int limit)
  {
    if (limit > job.n) limit = job.n;
    for (int k = job.next; k < limit;) {
      if (!job.next.compare_exchange_weak(k, k + 1)) continue;
      (*job.f)(k);
      ++job.helped;
      return true;
    }
    return false;
  }
  void finish(Job& job)
  {
    const int mine = job.helped + drain(job);
    std::unique_lock<std::mutex> lock(mu_);
    job.done += mine;
    job_ = nullptr;  // no thread takes it from here on
    done_cv_.wait(lock, [&] { return job.done == job.n && job.users == 0; });
  }
  int workers() const { return static_cast<int>(threads_.size()); }

 private:
  static int drain(Job& j)
  {
    int k, count = 0;
    while ((k = j.next.fetch_add(1)) < j.n) {
      (*j.f)(k);
      ++count;
    }
    return count;
  }
  void loop()
  {
    unsigned long long seen = 0;
    for (;;) {
      Job* j = nullptr;
      {
        std::unique_lock<std::mutex> lock(mu_);
        cv_.wait(lock, [&] { return stop_ || gen_ != seen; });
        if (stop_) return;
        seen = gen_;
        j = job_;
        if (!j) continue;
        ++j->users;
      }
      const int count = drain(*j);
      std::lock_guard<std::mutex> lock(mu_);
      j->done += count;
      --j->users;
      if (j->done == j->n && j->users == 0) done_cv_.notify_all();
    }
  }
  std::vector<std::thread> threads_;
  std::mutex mu_;
  std::condition_variable cv_, done_cv_;
  Job* job_ = nullptr;
  unsigned long long gen_ = 0;
  bool stop_ = false;
};
