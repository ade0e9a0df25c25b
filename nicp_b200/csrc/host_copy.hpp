// host_copy.hpp -- device -> host copies: straight into page-locked memory, into
// pageable memory through a context's own pinned slots.
//
// A copy into pageable memory that is handed to the driver waits for each of
// its staging transfers, and memory that the caller has just allocated is first
// touched -- a page fault every 4 KB -- by that same thread.  Here the slots'
// transfers overlap the copies into the caller's memory, and worker threads
// share those of a large one: a hand-written step at 320x240 (six copies of 75
// to 600 KB) 731 -> 502 us, a 640x480 cloud (32 MB) 12.1 -> 5.5 ms.  Waking
// the workers takes some 100 us, so smaller copies stay with the calling thread
// (2.4 MB: 0.92 ms alone, 1.09 shared).  Uploads stay with the driver: through
// the slots they were no faster from one thread, and slower shared.
//
// A page-locked destination takes one transfer and no copy after it: a 640x480
// projection's two images 213 us through the slots, 90 direct, a whole cloud of
// that size (32 MB) 2.2 ms through the slots, 0.63 direct.
//
// The slots (kSlots x kSlotBytes, allocated on first use) and the workers
// (started by the first copy of kShareBytes or more) belong to one context,
// are used by the one host thread that uses the context, and end with it.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <condition_variable>
#include <cstring>
#include <initializer_list>
#include <mutex>
#include <thread>
#include <vector>

namespace nicp {

class HostCopier {
 public:
  static constexpr size_t kSlotBytes = (size_t)1 << 20;
  static constexpr int kSlots = 8;
  static constexpr size_t kShareBytes = (size_t)8 << 20;
  static constexpr int kWorkers = 4;

  HostCopier() = default;
  HostCopier(const HostCopier &) = delete;
  HostCopier &operator=(const HostCopier &) = delete;
  // (the context's device is current, its streams are idle)
  ~HostCopier() {
    if (!workers_.empty()) {
      {
        std::lock_guard<std::mutex> l(m_);
        stop_ = true;
      }
      work_.notify_all();
      for (std::thread &t : workers_) t.join();
    }
    for (int k = 0; k < made_; k++) cudaEventDestroy(slots_[k].ev);
    if (mem_) cudaFreeHost(mem_);
  }

  // What a destination is.  (Both ends are looked up: a buffer of which only a
  // part is page-locked is pageable.)
  enum Kind { kPageable, kLocked, kDevice };
  static Kind kind(const void *dst, size_t bytes) {
    Kind k = kLocked;
    for (const char *p : {(const char *)dst, (const char *)dst + (bytes ? bytes - 1 : 0)}) {
      cudaPointerAttributes at = {};
      if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        cudaGetLastError();
        return kPageable;
      }
      if (at.type == cudaMemoryTypeUnregistered) return kPageable;
      if (at.type == cudaMemoryTypeDevice) k = kDevice;
    }
    return k;
  }

  // Device -> host, complete on return.  The stream's earlier work is waited for.
  struct Part {
    void *dst;
    const void *src;
    size_t bytes;
  };
  cudaError_t down(const Part *parts, int n, cudaStream_t s) {  // n <= 64
    size_t total = 0;         // bytes for the slots
    unsigned long long slow = 0;  // their parts
    cudaError_t e = cudaSuccess;
    for (int i = 0; i < n; i++) {
      const Part &p = parts[i];
      if (!p.dst || !p.bytes) continue;
      const Kind k = kind(p.dst, p.bytes);
      if (k == kDevice) e = cudaErrorInvalidValue;  // (not host memory: refused)
      if (k == kLocked && e == cudaSuccess) {
        // one transfer, no copy after it; where the runtime refuses (a range
        // that was page-locked in pieces) the slots do it
        if (cudaMemcpyAsync(p.dst, p.src, p.bytes, cudaMemcpyDeviceToHost, s) == cudaSuccess) continue;
        cudaGetLastError();
      }
      total += p.bytes;
      slow |= 1ull << i;
    }
    if (total && e == cudaSuccess && ready() != cudaSuccess) {
      // no page-locked memory for the slots: the driver's own staging
      cudaGetLastError();
      for (int i = 0; i < n && e == cudaSuccess; i++)
        if ((slow >> i) & 1) e = cudaMemcpyAsync(parts[i].dst, parts[i].src, parts[i].bytes, cudaMemcpyDeviceToHost, s);
      total = 0;
    }
    if (!total || e != cudaSuccess) {
      const cudaError_t err = cudaStreamSynchronize(s);
      return e != cudaSuccess ? e : err;
    }
    const bool share = total >= kShareBytes && start();
    Ring<Piece> flight;  // transfers on their way, in stream order
    auto land = [&] {    // the oldest transfer: wait, then copy out
      const Piece p = flight.pop();
      const cudaError_t err = cudaEventSynchronize(slots_[p.slot].ev);
      if (err == cudaSuccess) {
        if (share) submit(Job{p.host, slots_[p.slot].p, p.bytes, p.slot});
        else std::memcpy(p.host, slots_[p.slot].p, p.bytes);
      }
      return err;
    };
    int next = 0;
    for (int i = 0; i < n && e == cudaSuccess; i++) {
      if (!((slow >> i) & 1)) continue;
      for (size_t at = 0; at < parts[i].bytes && e == cudaSuccess;) {
        const size_t bytes = std::min(kSlotBytes, parts[i].bytes - at);
        if (flight.size == kSlots) e = land();
        if (e != cudaSuccess) break;
        const int k = next;
        next = (next + 1) % kSlots;
        if (share) wait_job(k);
        e = cudaMemcpyAsync(slots_[k].p, (const char *)parts[i].src + at, bytes, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaEventRecord(slots_[k].ev, s);
        if (e == cudaSuccess) flight.push(Piece{(char *)parts[i].dst + at, bytes, k});
        at += bytes;
      }
    }
    while (flight.size) {
      const cudaError_t err = land();
      if (e == cudaSuccess) e = err;
    }
    if (share) drain();
    const cudaError_t err = cudaStreamSynchronize(s);
    return e != cudaSuccess ? e : err;
  }

 private:
  struct Slot {
    char *p = nullptr;
    cudaEvent_t ev = nullptr;
    bool job = false;  // a worker copies from it (under m_)
  };
  // At most kSlots of anything: a slot has one transfer, then one job.  (Nothing
  // here allocates once the slots and workers exist, so a copy under way cannot
  // end in an exception that leaves jobs writing to the caller's memory.)
  template <class T>
  struct Ring {
    T at[kSlots];
    int first = 0, size = 0;
    void push(const T &v) { at[(first + size++) % kSlots] = v; }
    T pop() {
      const T v = at[first];
      first = (first + 1) % kSlots;
      size--;
      return v;
    }
  };
  struct Piece {
    char *host;
    size_t bytes;
    int slot;
  };
  struct Job {
    void *dst;
    const void *src;
    size_t bytes;
    int slot;
  };

  cudaError_t ready() {
    if (mem_ && made_ == kSlots) return cudaSuccess;
    cudaError_t e = cudaSuccess;
    if (!mem_ && (e = cudaMallocHost(&mem_, kSlots * kSlotBytes)) != cudaSuccess) {
      mem_ = nullptr;
      return e;
    }
    for (; made_ < kSlots; made_++) {
      if ((e = cudaEventCreateWithFlags(&slots_[made_].ev, cudaEventDisableTiming)) != cudaSuccess) return e;
      slots_[made_].p = mem_ + made_ * kSlotBytes;
    }
    return cudaSuccess;
  }
  // The workers, if threads can be had (else the calling thread copies alone).
  bool start() {
    if (!workers_.empty()) return true;
    const int n = std::min<int>(kWorkers, (int)std::thread::hardware_concurrency() - 1);
    try {
      workers_.reserve(std::max(n, 0));
      for (int k = 0; k < n; k++) workers_.emplace_back([this] { work(); });
    } catch (...) {
    }
    return !workers_.empty();
  }
  void work() {
    std::unique_lock<std::mutex> l(m_);
    for (;;) {
      work_.wait(l, [&] { return stop_ || jobs_.size; });
      if (!jobs_.size) return;
      one(l);
    }
  }
  void one(std::unique_lock<std::mutex> &l) {
    const Job j = jobs_.pop();
    l.unlock();
    std::memcpy(j.dst, j.src, j.bytes);
    l.lock();
    slots_[j.slot].job = false;
    pending_--;
    done_.notify_all();
  }
  void submit(const Job &j) {
    {
      std::lock_guard<std::mutex> l(m_);
      slots_[j.slot].job = true;
      pending_++;
      jobs_.push(j);
    }
    work_.notify_one();
  }
  // The calling thread takes jobs too while it waits.
  void wait_job(int slot) {
    std::unique_lock<std::mutex> l(m_);
    while (slots_[slot].job) {
      if (jobs_.size) one(l);
      else done_.wait(l, [&] { return !slots_[slot].job || jobs_.size; });
    }
  }
  void drain() {
    std::unique_lock<std::mutex> l(m_);
    while (pending_) {
      if (jobs_.size) one(l);
      else done_.wait(l, [&] { return !pending_ || jobs_.size; });
    }
  }
  char *mem_ = nullptr;
  Slot slots_[kSlots];
  int made_ = 0;
  std::vector<std::thread> workers_;
  std::mutex m_;
  std::condition_variable work_, done_;
  Ring<Job> jobs_;
  int pending_ = 0;
  bool stop_ = false;
};

}  // namespace nicp
