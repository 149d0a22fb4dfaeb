// hostcopy.cuh -- large results from the device into pageable host arrays, by a
// few host threads through a small pinned ring.
//
// A pageable copy is one thread's: the driver's copy out of its own staging,
// and for a result array that the caller has just allocated also the page
// faults of its first touch, which take most of the time (52 MB: 11.7 ms into
// fresh pages, 3.2 ms into touched ones; the link needs 1.0).  Here up to
// kWorkers threads touch the pages (MADV_POPULATE_WRITE: contents stay) while the
// kernels still run, sleep until the first chunk is there, then move chunks from
// the ring to the array, the copies staying on the caller's stream in order: 52 MB
// fresh 2.8 ms, and the page touching overlaps the kernels.  Below kStagedMin a
// plain copy is as quick; arrays the caller has pinned are copied directly.  (The
// other way, chunks written by several threads read back over the link at half the
// rate of the driver's own staging: inputs are copied plainly.)
//
// The ring (6 MB) and the threads are the process's, one set per device, shared
// by its contexts and gone with the last of them that used it.  One call uses
// them at a time; another one meanwhile copies plainly.  They take 3 to 10 ms to
// make (nearly all of it the pinning), which is what they save on some 30 MB: so
// the first kPlainFirst bytes are copied plainly, and a program that has one window
// to copy pays nothing for them.
#pragma once
#include <cuda_runtime.h>
#include <sys/mman.h>
#include <unistd.h>

#include <atomic>
#include <condition_variable>
#include <cstdint>
#include <algorithm>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

namespace atlasgpu {

struct CopySeg {
  void* host;
  const void* dev;
  size_t bytes;
};

constexpr size_t kStagedMin = 8 << 20;    // bytes of a call's large arrays from which the threads are used (below:
                                          // under 1 ms a call)
constexpr size_t kPlainFirst = 32 << 20;  // bytes of such calls copied plainly before the ring and the threads are made
constexpr size_t kStagedSeg = 256 << 10;  // smaller arrays of the same call are copied plainly

class HostCopier {
 public:
  explicit HostCopier(int device) : device_(device), pid_(getpid()) {}
  ~HostCopier() {
    {
      std::lock_guard<std::mutex> l(m_);
      quit_ = true;
    }
    cv_.notify_all();
    for (auto& t : threads_) {
      if (pid_ == getpid()) t.join();
      else t.detach();  // a forked child has no such threads
    }
    for (int i = 0; i < nev_; ++i) {
      cudaEventSynchronize(ev_[i]);
      cudaEventDestroy(ev_[i]);
    }
    if (pin_) cudaFreeHost(pin_);
  }

  // the process's copier for a device
  static std::shared_ptr<HostCopier> of(int device) {
    static std::mutex m;
    static std::map<int, std::weak_ptr<HostCopier>> all;
    std::lock_guard<std::mutex> l(m);
    std::shared_ptr<HostCopier> c = all[device].lock();
    if (!c) all[device] = c = std::make_shared<HostCopier>(device);
    return c;
  }

  // Device to host, complete on return, the outcome in *e; false: nothing done,
  // the caller copies plainly (another call is using the ring, or there is none).
  bool out(cudaStream_t s, const std::vector<CopySeg>& segs, size_t bytes, cudaError_t* e) {
    std::unique_lock<std::mutex> use(use_, std::try_to_lock);
    if (!use || pid_ != getpid() || !ready(bytes)) return false;
    *e = run(s, segs);
    return true;
  }

 private:
  bool ready(size_t bytes) {
    if (pin_) return true;
    if (failed_) return false;
    if (plain_ < kPlainFirst) {
      plain_ += bytes;
      return false;
    }
    failed_ = true;
    for (; nev_ < kSlots; ++nev_)
      if (cudaEventCreateWithFlags(&ev_[nev_], cudaEventDisableTiming) != cudaSuccess) {
        cudaGetLastError();
        return false;
      }
    void* p = nullptr;
    if (cudaMallocHost(&p, kSlots * kChunk) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    pin_ = (char*)p;
    const int want = std::min<int>(kWorkers, (int)std::thread::hardware_concurrency() / 2 - 1);
    try {
      for (int i = 0; i < want; ++i) threads_.emplace_back([this, i] { worker(i); });
    } catch (...) {
      // as many as there are; with none the calling thread does it all
    }
    failed_ = false;
    return true;
  }

  cudaError_t issue(cudaStream_t s, int k) {
    const int sl = k % kSlots;
    const Chunk& c = chunks_[k];
    cudaError_t e = cudaMemcpyAsync(pin_ + (size_t)sl * kChunk, c.dev, c.bytes, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaEventRecord(ev_[sl], s);
    return e;
  }

  cudaError_t run(cudaStream_t s, const std::vector<CopySeg>& segs) {
    cut(segs);
    const int n = (int)chunks_.size(), first = std::min(n, kSlots);
    cudaError_t e = cudaSuccess;
    for (int k = 0; k < first && e == cudaSuccess; ++k) {
      e = cudaEventSynchronize(ev_[k]);  // a copy into the slot that an earlier call gave up on
      if (e == cudaSuccess) e = issue(s, k);
    }
    if (e != cudaSuccess) return e;
    open(first);
    touch_pages();
    e = cudaEventSynchronize(ev_[0]);  // the kernels: one thread waits for them, as in a plain copy
    if (e == cudaSuccess) copying();
    for (int k = kSlots; k < n && e == cudaSuccess && !abort_; ++k) {
      while (done_[k % kSlots].load(std::memory_order_acquire) != k - kSlots && !abort_)
        if (!take_out()) std::this_thread::yield();
      if (!abort_) e = issue(s, k);
      if (!abort_ && e == cudaSuccess) issued_.store(k + 1, std::memory_order_release);
    }
    if (e != cudaSuccess) abort_ = true;
    while (!abort_ && take_out()) {
    }
    close();
    return e != cudaSuccess ? e : err_;
  }

  static constexpr size_t kChunk = 512 << 10;
  static constexpr size_t kTouch = 2 << 20;
  static constexpr int kSlots = 12, kWorkers = 7;
  struct Chunk {
    char *host, *dev;
    size_t bytes;
  };

  void cut(const std::vector<CopySeg>& segs) {
    chunks_.clear();
    touch_.clear();
    for (const CopySeg& q : segs) {
      for (size_t o = 0; o < q.bytes; o += kChunk)
        chunks_.push_back(Chunk{(char*)q.host + o, (char*)q.dev + o, std::min(kChunk, q.bytes - o)});
      for (size_t o = 0; o < q.bytes; o += kTouch)
        touch_.push_back(Chunk{(char*)q.host + o, nullptr, std::min(kTouch, q.bytes - o)});
    }
  }

  void open(int issued) {
    for (auto& d : done_) d.store(-1, std::memory_order_relaxed);
    ticket_ = touched_ = 0;
    issued_ = issued;
    abort_ = false;
    err_ = cudaSuccess;
    {
      std::lock_guard<std::mutex> l(m_);
      job_ = true;
      copying_ = false;
      want_ = (int)std::min(threads_.size(), chunks_.size() / 2);
      ++gen_;
    }
    if (want_) cv_.notify_all();
  }
  // the first chunk is there
  void copying() {
    {
      std::lock_guard<std::mutex> l(m_);
      copying_ = true;
    }
    if (want_) cv_.notify_all();
  }
  // no worker is in the job after this
  void close() {
    std::unique_lock<std::mutex> l(m_);
    job_ = false;
    if (!copying_) cv_.notify_all();
    idle_.wait(l, [this] { return running_ == 0; });
  }

  void worker(int id) {
    cudaSetDevice(device_);
    uint64_t seen = 0;
    std::unique_lock<std::mutex> l(m_);
    for (;;) {
      cv_.wait(l, [&] { return quit_ || gen_ != seen; });
      if (quit_) return;
      seen = gen_;
      if (!job_ || id >= want_) continue;
      ++running_;
      l.unlock();
      const int n = (int)chunks_.size();
      touch_pages();
      l.lock();
      cv_.wait(l, [this] { return copying_ || !job_; });
      l.unlock();
      for (int k; !abort_ && (k = ticket_.fetch_add(1)) < n;) {
        while (issued_.load(std::memory_order_acquire) <= k && !abort_) std::this_thread::yield();
        if (!abort_) copy_out(k);
      }
      l.lock();
      if (--running_ == 0) idle_.notify_all();
    }
  }

  // the calling thread takes a chunk that needs no wait for itself
  bool take_out() {
    int t = ticket_.load();
    if (t >= issued_.load() || !ticket_.compare_exchange_strong(t, t + 1)) return false;
    copy_out(t);
    return true;
  }
  void copy_out(int k) {
    const int sl = k % kSlots;
    if (!wait_event(sl)) return;
    memcpy(chunks_[k].host, pin_ + (size_t)sl * kChunk, chunks_[k].bytes);
    done_[sl].store(k, std::memory_order_release);
  }
  bool wait_event(int sl) {
    const cudaError_t e = cudaEventSynchronize(ev_[sl]);
    if (e == cudaSuccess) return true;
    std::lock_guard<std::mutex> l(m_);
    err_ = e;
    abort_ = true;
    return false;
  }
  // whole pages inside the arrays; a kernel without the call leaves them to the copies
  void touch_pages() {
#ifndef MADV_POPULATE_WRITE
#define MADV_POPULATE_WRITE 23
#endif
    const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE);
    for (size_t k; (k = (size_t)touched_.fetch_add(1)) < touch_.size();) {
      const uintptr_t a = ((uintptr_t)touch_[k].host + page - 1) / page * page;
      const uintptr_t b = ((uintptr_t)touch_[k].host + touch_[k].bytes) / page * page;
      if (b > a) (void)madvise((void*)a, b - a, MADV_POPULATE_WRITE);
    }
  }

  int device_;
  pid_t pid_;
  std::mutex use_;      // held by the call that uses the rest
  size_t plain_ = 0;    // bytes copied plainly before there was a ring
  char* pin_ = nullptr;
  bool failed_ = false;
  int nev_ = 0;
  cudaEvent_t ev_[kSlots] = {};
  std::vector<std::thread> threads_;
  std::mutex m_;
  std::condition_variable cv_, idle_;
  uint64_t gen_ = 0;
  bool quit_ = false;
  bool job_ = false, copying_ = false;
  int want_ = 0, running_ = 0;
  std::vector<Chunk> chunks_, touch_;
  std::atomic<int> done_[kSlots];
  std::atomic<int> issued_{0}, ticket_{0}, touched_{0};
  std::atomic<bool> abort_{false};
  cudaError_t err_ = cudaSuccess;
};

}  // namespace atlasgpu
