// Host copies split over threads (the server's request copies).
#pragma once

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstdint>
#include <cstring>
#include <memory>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

namespace rfmm {

// Host copies of a request's bodies, split over the calling thread and a few
// helpers: one thread copies about 14 GB/s (10 into memory it touches for the
// first time), a twentieth of the host link and less than the GPU steps
// through, so a burst of requests was bound by its submit and result copies.
// A copy is cut into pieces that the caller and the helpers take in turn; the
// caller never waits for a helper to wake, only for pieces already taken.
// Any number of threads may copy at once.  copy() and start() throw nothing:
// without memory for a job or threads for helpers the caller copies alone.
class CopyPool {
 public:
  ~CopyPool() {
    {
      std::lock_guard<std::mutex> lk(m_);
      stop_ = true;
    }
    cv_.notify_all();
    for (auto &t : helpers_) t.join();
  }
  void start(unsigned helpers) {
    try {
      for (unsigned i = 0; i < helpers; i++) helpers_.emplace_back(&CopyPool::loop, this);
    } catch (...) {  // no more threads to be had: the callers copy alone
    }
  }
  void copy(void *dst, const void *src, size_t bytes) {
    if (bytes < 4 * kPiece || helpers_.empty()) {
      std::memcpy(dst, src, bytes);
      return;
    }
    std::shared_ptr<Job> job;
    try {
      job = std::make_shared<Job>();
      job->dst = static_cast<uint8_t *>(dst);
      job->src = static_cast<const uint8_t *>(src);
      job->bytes = bytes;
      job->pieces = (bytes + kPiece - 1) / kPiece;
      std::lock_guard<std::mutex> lk(m_);
      jobs_.push_back(job);
    } catch (const std::bad_alloc &) {
      std::memcpy(dst, src, bytes);
      return;
    }
    cv_.notify_all();
    work(*job);
    std::unique_lock<std::mutex> lk(m_);
    jobs_.erase(std::find(jobs_.begin(), jobs_.end(), job));
    done_cv_.wait(lk, [&] { return job->done == job->pieces; });
  }

 private:
  static constexpr size_t kPiece = 256u << 10;
  struct Job {
    uint8_t *dst = nullptr;
    const uint8_t *src = nullptr;
    size_t bytes = 0, pieces = 0;
    std::atomic<size_t> next{0};
    size_t done = 0;  // under m_
  };
  void work(Job &j) {
    size_t mine = 0;
    for (size_t i; (i = j.next.fetch_add(1)) < j.pieces; mine++) {
      const size_t at = i * kPiece;
      std::memcpy(j.dst + at, j.src + at, std::min(kPiece, j.bytes - at));
    }
    if (mine == 0) return;
    std::lock_guard<std::mutex> lk(m_);
    j.done += mine;
    if (j.done == j.pieces) done_cv_.notify_all();
  }
  void loop() {
    std::unique_lock<std::mutex> lk(m_);
    for (;;) {
      std::shared_ptr<Job> job;
      cv_.wait(lk, [&] {
        if (stop_) return true;
        for (auto &j : jobs_)
          if (j->next.load() < j->pieces) {
            job = j;
            return true;
          }
        return false;
      });
      if (stop_) return;
      lk.unlock();
      work(*job);
      lk.lock();
    }
  }
  std::vector<std::thread> helpers_;
  std::vector<std::shared_ptr<Job>> jobs_;
  std::mutex m_;
  std::condition_variable cv_, done_cv_;
  bool stop_ = false;
};

}  // namespace rfmm
