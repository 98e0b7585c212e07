// Page-locked staging buffers and copy threads, shared by every handle of the process.
//
// Pageable memory reaches the GPU through the driver's own bounce buffer at 10-12 GB/s on one host thread, and a
// result array fresh from the allocator costs a page fault every 4 KB on top: a 100 000-query, top-100 search spent
// 22 of its 29 ms there.  Here several threads copy between the caller's memory and page-locked buffers while the GPU
// works on the buffers before and after.
//
// Bounded: at most kMaxBuffers buffers of kBufferBytes, allocated as they are asked for, and kMaxThreads threads.  All
// of it is given back when the last handle is destroyed.  Any number of threads may use it at once.
#pragma once
#include <cuda_runtime.h>
#include <pthread.h>

#include <algorithm>
#include <condition_variable>
#include <cstring>
#include <deque>
#include <functional>
#include <memory>
#include <mutex>
#include <new>
#include <system_error>
#include <thread>
#include <vector>

namespace hnsw {

class HostStage {
 public:
  // 2 / 4 / 8 MB: 17.6 / 12.3 / 10.5 ms for that search, 12.9 / 17 / 7.5 ms for loading a 132 MB index file
  static constexpr size_t kBufferBytes = 8u << 20;
  static constexpr int kMaxBuffers = 8;
  static constexpr int kMaxThreads = 8;
  static constexpr size_t kShareBytes = 256u << 10;  // below this a copy is not worth waking another thread

  // (never destroyed: handles that outlive main() may still use it)
  static HostStage& Get() {
    static HostStage* one = [] {
      auto* stage = new HostStage;
      pthread_atfork([] { Get().mu_.lock(); }, [] { Get().mu_.unlock(); }, [] { Get().Forked(); });
      return stage;
    }();
    return *one;
  }

  void AddUser() {
    std::lock_guard<std::mutex> lock(mu_);
    ++users_;
  }
  void DropUser() {
    std::vector<std::thread> threads;
    {
      std::lock_guard<std::mutex> lock(mu_);
      if (--users_ > 0) return;
      for (void* p : free_) cudaFreeHost(p);
      made_ -= (int)free_.size();
      free_.clear();
      ++generation_;
      threads.swap(threads_);
    }
    work_.notify_all();
    for (std::thread& t : threads) t.join();
  }

  // A buffer, or nullptr: page-locked memory cannot be had, or all buffers are in use.  Nobody waits for one: the others
  // may be held for as long as somebody's file takes to write, and every transfer has another way.
  void* Acquire() {
    {
      std::lock_guard<std::mutex> lock(mu_);
      if (!free_.empty()) {
        void* p = free_.back();
        free_.pop_back();
        return p;
      }
      if (made_ >= kMaxBuffers) return nullptr;
      ++made_;
    }
    void* p = nullptr;
    if (cudaHostAlloc(&p, kBufferBytes, cudaHostAllocPortable) == cudaSuccess) return p;
    cudaGetLastError();
    std::lock_guard<std::mutex> lock(mu_);
    --made_;
    return nullptr;
  }
  void Release(void* p) {
    if (!p) return;
    std::lock_guard<std::mutex> lock(mu_);
    free_.push_back(p);
  }

  // f(0) ... f(n - 1) on the calling thread and the pool's; returns when all are done.  f must not throw.
  void ParallelFor(int n, const std::function<void(int)>& f) {
    if (n <= 1) {
      if (n == 1) f(0);
      return;
    }
    auto job = std::make_shared<Job>();
    job->f = &f;
    job->n = n;
    {
      std::lock_guard<std::mutex> lock(mu_);
      const int want = std::min({n - 1, kMaxThreads, (int)std::thread::hardware_concurrency() - 1});
      try {
        while ((int)threads_.size() < want) threads_.emplace_back([this, mine = generation_] { Serve(mine); });
      } catch (const std::system_error&) {
        // the process is at its limit of threads: the calling thread and those there are do the work
      }
      jobs_.push_back(job);
    }
    work_.notify_all();
    Run(*job);
    std::unique_lock<std::mutex> lock(mu_);
    job->over.wait(lock, [&] { return job->done == job->n; });
    for (auto it = jobs_.begin(); it != jobs_.end(); ++it)
      if (*it == job) {
        jobs_.erase(it);
        break;
      }
  }
  void Copy(void* dst, const void* src, size_t bytes) {
    const size_t part = std::max(kShareBytes, (bytes / (kMaxThreads + 1) + 4095) / 4096 * 4096);
    ParallelFor((int)((bytes + part - 1) / part), [&](int i) {
      const size_t lo = (size_t)i * part;
      std::memcpy(static_cast<char*>(dst) + lo, static_cast<const char*>(src) + lo, std::min(part, bytes - lo));
    });
  }

 private:
  struct Job {
    const std::function<void(int)>* f;
    int n, next = 0, done = 0;  // under mu_
    std::condition_variable over;
  };
  // takes parts of the job until none is left
  void Run(Job& job) {
    std::unique_lock<std::mutex> lock(mu_);
    while (job.next < job.n) {
      const int i = job.next++;
      lock.unlock();
      (*job.f)(i);
      lock.lock();
      if (++job.done == job.n) job.over.notify_all();
    }
  }
  // until the users that this thread was started for are gone; others may have come and gone since
  void Serve(long long mine) {
    std::unique_lock<std::mutex> lock(mu_);
    while (mine == generation_) {
      std::shared_ptr<Job> job;
      for (auto& j : jobs_)
        if (j->next < j->n) {
          job = j;
          break;
        }
      if (!job) {
        work_.wait(lock);
        continue;
      }
      lock.unlock();
      Run(*job);
      lock.lock();
    }
  }

  // In a forked child: the threads are not there, so nobody may wait for them, or on what they waited on.  Their objects
  // are left behind (a destructor would wait).
  void Forked() {
    new (&threads_) std::vector<std::thread>;
    new (&jobs_) std::deque<std::shared_ptr<Job>>;
    new (&work_) std::condition_variable;
    ++generation_;
    mu_.unlock();
  }

  std::mutex mu_;
  std::condition_variable work_;
  std::vector<void*> free_;
  std::vector<std::thread> threads_;
  std::deque<std::shared_ptr<Job>> jobs_;
  int users_ = 0, made_ = 0;
  long long generation_ = 0;  // counts the times the last user went
};

// A buffer of the stage for the lifetime of a scope.
class StageBuffer {
 public:
  StageBuffer() : p_(HostStage::Get().Acquire()) {}
  ~StageBuffer() { HostStage::Get().Release(p_); }
  StageBuffer(const StageBuffer&) = delete;
  StageBuffer& operator=(const StageBuffer&) = delete;
  unsigned char* get() const { return static_cast<unsigned char*>(p_); }

 private:
  void* p_;
};

// A staging buffer that the work of a stream reads and writes: it goes back when that work is over, also when an
// exception takes the scope down.
class StreamBuffer {
 public:
  StreamBuffer() = default;
  StreamBuffer(const StreamBuffer&) = delete;
  StreamBuffer& operator=(const StreamBuffer&) = delete;
  ~StreamBuffer() { Wait(); }
  // false: none to be had
  bool Open() {
    buffer_.reset(new StageBuffer);
    if (!buffer_->get()) buffer_.reset();
    return buffer_ != nullptr;
  }
  unsigned char* get() const { return buffer_->get(); }
  // from here on `stream` may have work on the buffer
  void Use(cudaStream_t stream) {
    stream_ = stream;
    busy_ = true;
  }
  cudaError_t Wait() {
    if (!busy_) return cudaSuccess;
    busy_ = false;
    return cudaStreamSynchronize(stream_);
  }

 private:
  std::unique_ptr<StageBuffer> buffer_;
  cudaStream_t stream_ = nullptr;
  bool busy_ = false;
};

// A ring of staging buffers for a transfer in pieces: fill or drain one while the device works on the others.
class Pipeline {
 public:
  static constexpr int kDepth = 3;
  class Slot {
   public:
    unsigned char* host() const { return buffer_->get(); }

   private:
    friend class Pipeline;
    std::unique_ptr<StageBuffer> buffer_;
    cudaEvent_t done_ = nullptr;
    bool pending_ = false;
  };
  Pipeline() = default;
  Pipeline(const Pipeline&) = delete;
  Pipeline& operator=(const Pipeline&) = delete;
  // the device is through with every buffer before it goes back
  ~Pipeline() {
    for (Slot& s : slots_) {
      if (s.pending_) cudaEventSynchronize(s.done_);
      if (s.done_) cudaEventDestroy(s.done_);
    }
  }
  // buffers for `pieces` pieces (at most kDepth); false: none to be had
  bool Open(long long pieces) {
    for (; depth_ < kDepth && depth_ < pieces; ++depth_) {
      Slot& s = slots_[depth_];
      s.buffer_.reset(new StageBuffer);
      if (!s.buffer_->get() || cudaEventCreateWithFlags(&s.done_, cudaEventDisableTiming) != cudaSuccess) {
        s.buffer_.reset();
        cudaGetLastError();
        break;
      }
    }
    return depth_ > 0;
  }
  int depth() const { return depth_; }
  Slot& At(long long i) { return slots_[i % depth_]; }
  Slot& Next() { return At(turn_++); }
  cudaError_t Mark(Slot& s, cudaStream_t stream) {
    s.pending_ = true;
    return cudaEventRecord(s.done_, stream);
  }
  cudaError_t Wait(Slot& s) {
    if (!s.pending_) return cudaSuccess;
    s.pending_ = false;
    return cudaEventSynchronize(s.done_);
  }

 private:
  Slot slots_[kDepth];
  int depth_ = 0;
  long long turn_ = 0;
};

}  // namespace hnsw
