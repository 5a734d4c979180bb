// Copies between pageable host memory and the device for calls whose operands live there.
//
// The driver moves pageable memory through a staging buffer of its own, one thread copying, and
// a download holds the calling thread until it is complete: 1024^3 u8 x s8 with beta = 1
// (6 MB up, 4 MB down) took 720 us.  Here a few threads share each piece's copy into
// (or out of) a ring of pinned slots, the bus transfers of the pieces before it run meanwhile, and a
// download's last copy is left until the call has issued everything else: 410 us (five threads 390, but
// then one of them more often has no core when its piece is waited for).
#pragma once

#include <cuda_runtime.h>
#include <dlfcn.h>
#include <pthread.h>
#include <signal.h>
#if defined(__x86_64__)
#include <immintrin.h>
#endif

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <thread>

namespace {

inline void spin_pause() {
#if defined(__x86_64__)
  _mm_pause();
#elif defined(__aarch64__)
  asm volatile("yield" ::: "memory");
#endif
}

// `rows` rows of `width` bytes.
struct RowCopy {
  uint8_t* dst;
  const uint8_t* src;
  size_t dst_pitch, src_pitch, width, rows;
  // the part-th of `parts` equal shares: of the bytes when the rows are contiguous, else of the rows
  void share(size_t part, size_t parts) const {
    if (dst_pitch == width && src_pitch == width) {
      const size_t total = width * rows, step = ((total + parts - 1) / parts + 63) / 64 * 64;
      const size_t begin = std::min(total, part * step), end = std::min(total, begin + step);
      if (end > begin) std::memcpy(dst + begin, src + begin, end - begin);
      return;
    }
    for (size_t r = part * rows / parts; r < (part + 1) * rows / parts; ++r)
      std::memcpy(dst + r * dst_pitch, src + r * src_pitch, width);
  }
};

// A few threads that share one copy at a time with the thread that asks for it, in pieces of
// about 64 KB that each of them takes when it is free: a thread that gets no core (torch's own
// threads may be spinning on them all) delays nobody, where equal shares made calls wait a
// scheduler's slice of 4 ms for it.  The threads are started by the first large copy of the
// process, watch for the next copy for 200 us after each (a call's pieces follow one another
// within microseconds), sleep otherwise, and end with the process (detached: nothing joins
// them, in a forked child neither).  So that nobody else has to know of them, they take none of the
// process's signals, and the shared library that holds their code is kept mapped when the
// program closes it.  A caller that finds them busy with another caller's copy
// does its own alone.
class CopyThreads {
 public:
  static constexpr int kThreads = 3;

  void copy(const RowCopy& c) {
    const size_t bytes = c.width * c.rows;
    std::unique_lock<std::mutex> mine(owner_mu_, std::defer_lock);
    if (bytes < (128u << 10) || !mine.try_lock()) {
      c.share(0, 1);
      return;
    }
    if (!started_) start();
    const uint32_t parts = static_cast<uint32_t>(std::min<size_t>(1024, (bytes + (64u << 10) - 1) / (64u << 10)));
    job_ = c;
    done_.store(0, std::memory_order_relaxed);
    ticket_.store(make_ticket(++job_number_, parts, 0));  // (a sleeper that misses this only helps less)
    if (sleepers_.load() > 0) wake_.notify_all();
    while (take_part()) {
    }
    while (done_.load(std::memory_order_acquire) < parts) spin_pause();
  }

 private:
  // The job's number (so that a late thread cannot take a part of one job for another's), how
  // many parts it has, and the next one to be taken.
  static uint64_t make_ticket(uint32_t number, uint32_t parts, uint32_t next) {
    return static_cast<uint64_t>(number) << 32 | parts << 16 | next;
  }
  static bool has_work(uint64_t t) { return (t & 0xFFFF) < (t >> 16 & 0xFFFF); }

  // Takes and copies one part; false when none is left.  While a part is being copied its job
  // cannot end, so job_ is the ticket's.
  bool take_part() {
    uint64_t t = ticket_.load(std::memory_order_acquire);
    do {
      if (!has_work(t)) return false;
    } while (!ticket_.compare_exchange_weak(t, t + 1, std::memory_order_acq_rel, std::memory_order_acquire));
    job_.share(t & 0xFFFF, t >> 16 & 0xFFFF);
    done_.fetch_add(1, std::memory_order_release);
    return true;
  }

  void start() {
    started_ = true;
    Dl_info self;
    if (dladdr(reinterpret_cast<void*>(&spin_pause), &self) == 0 ||
        dlopen(self.dli_fname, RTLD_NOW | RTLD_NOLOAD | RTLD_NODELETE) == nullptr)
      return;  // (the callers copy alone)
    sigset_t all, callers;
    sigfillset(&all);
    if (pthread_sigmask(SIG_SETMASK, &all, &callers) != 0) return;
    const unsigned cores = std::thread::hardware_concurrency();
    const int n = std::max(0, std::min(kThreads, static_cast<int>(cores) / 2 - 1));
    try {
      for (int i = 0; i < n; ++i) std::thread([this] { run(); }).detach();
    } catch (...) {
      // no more threads to be had: the ones that exist share the work
    }
    pthread_sigmask(SIG_SETMASK, &callers, nullptr);
  }

  void run() {
    for (;;) {
      const auto until = std::chrono::steady_clock::now() + std::chrono::microseconds(200);
      bool found = false;
      for (int i = 0; !found; ++i) {
        found = take_part();
        if (found) break;
        spin_pause();
        if ((i & 63) == 63 && std::chrono::steady_clock::now() > until) break;
      }
      if (found) continue;
      std::unique_lock<std::mutex> lk(sleep_mu_);
      sleepers_.fetch_add(1);
      wake_.wait(lk, [&] { return has_work(ticket_.load()); });
      sleepers_.fetch_sub(1);
    }
  }

  std::mutex owner_mu_;  // held by the caller whose copy is being shared
  bool started_ = false;
  RowCopy job_{};
  uint32_t job_number_ = 0;
  std::atomic<uint64_t> ticket_{0};
  std::atomic<uint32_t> done_{0};
  std::atomic<int> sleepers_{0};
  std::mutex sleep_mu_;
  std::condition_variable wake_;
};

CopyThreads& copy_threads() {
  static CopyThreads* t = new CopyThreads;  // never destroyed: its threads outlive main()
  return *t;
}

// The pinned slots of one device (kSlots MB, allocated by the first large pageable copy).  Used
// under the device's lock.  A slot is busy while its transfer runs, and a download's until its
// bytes have also been copied out; taking a busy slot finishes it first.
class StagingRing {
 public:
  static constexpr int kSlots = 16;
  static constexpr size_t kSlotBytes = size_t{1} << 20;
  static constexpr size_t kSmallest = size_t{64} << 10;  // below this the driver's own path is as fast

  // Whether a copy of `bytes` at host address `host` on `stream` goes through the ring.
  bool serves(const void* host, size_t width, size_t bytes, cudaStream_t stream) {
    if (bytes < kSmallest || width > kSlotBytes) return false;
    cudaPointerAttributes attr;
    if (cudaPointerGetAttributes(&attr, host) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (attr.type != cudaMemoryTypeUnregistered || cudaStreamIsCapturing(stream, &cs) != cudaSuccess ||
        cs != cudaStreamCaptureStatusNone) {
      cudaGetLastError();
      return false;
    }
    return ready();
  }

  cudaError_t upload(void* dst, size_t dst_pitch, const void* src, size_t src_pitch, size_t width, size_t rows,
                     cudaStream_t stream) {
    for (size_t r0 = 0; r0 < rows;) {
      const size_t n = std::min(rows - r0, kSlotBytes / width);
      Slot* s = nullptr;
      if (cudaError_t e = take(&s)) return e;
      copy_threads().copy(RowCopy{s->mem, static_cast<const uint8_t*>(src) + r0 * src_pitch, width, src_pitch, width, n});
      uint8_t* to = static_cast<uint8_t*>(dst) + r0 * dst_pitch;
      if (cudaError_t e = cudaMemcpy2DAsync(to, dst_pitch, s->mem, width, width, n, cudaMemcpyHostToDevice, stream))
        return e;
      if (cudaError_t e = cudaEventRecord(s->done, stream)) return e;
      s->busy = true;
      r0 += n;
    }
    return cudaSuccess;
  }

  // Enqueues the transfer; the bytes are in place after finish().
  cudaError_t download(void* dst, size_t dst_pitch, const void* src, size_t src_pitch, size_t width, size_t rows,
                       cudaStream_t stream) {
    for (size_t r0 = 0; r0 < rows;) {
      const size_t n = std::min(rows - r0, kSlotBytes / width);
      Slot* s = nullptr;
      if (cudaError_t e = take(&s)) return e;
      const uint8_t* from = static_cast<const uint8_t*>(src) + r0 * src_pitch;
      if (cudaError_t e = cudaMemcpy2DAsync(s->mem, width, from, src_pitch, width, n, cudaMemcpyDeviceToHost, stream))
        return e;
      if (cudaError_t e = cudaEventRecord(s->done, stream)) return e;
      s->busy = true;
      s->out = RowCopy{static_cast<uint8_t*>(dst) + r0 * dst_pitch, s->mem, dst_pitch, width, width, n};
      r0 += n;
    }
    return cudaSuccess;
  }

  // Completes every download enqueued so far, oldest first.
  cudaError_t finish() {
    if (!slots_[0].mem) return cudaSuccess;
    for (int i = 0; i < kSlots; ++i) {
      Slot& s = slots_[(next_ + i) % kSlots];
      if (s.busy && s.out.rows > 0)
        if (cudaError_t e = settle(s)) return e;
    }
    return cudaSuccess;
  }

  // After a call that failed half way: waits for what is in flight and copies nothing out.
  void forget() {
    for (Slot& s : slots_) {
      if (s.busy && s.out.rows > 0 && cudaEventSynchronize(s.done) != cudaSuccess) cudaGetLastError();
      s.out.rows = 0;
    }
  }

 private:
  struct Slot {
    uint8_t* mem = nullptr;
    cudaEvent_t done = nullptr;
    bool busy = false;
    RowCopy out{};
  };

  cudaError_t settle(Slot& s) {
    if (cudaError_t e = cudaEventSynchronize(s.done)) return e;
    if (s.out.rows > 0) copy_threads().copy(s.out);
    s.out.rows = 0;
    s.busy = false;
    return cudaSuccess;
  }

  cudaError_t take(Slot** out) {
    Slot& s = slots_[next_];
    next_ = (next_ + 1) % kSlots;
    if (s.busy)
      if (cudaError_t e = settle(s)) return e;
    *out = &s;
    return cudaSuccess;
  }

  bool ready() {
    if (slots_[0].mem) return true;
    if (failed_) return false;
    void* mem = nullptr;
    failed_ = cudaHostAlloc(&mem, kSlots * kSlotBytes, cudaHostAllocDefault) != cudaSuccess;
    for (int i = 0; i < kSlots && !failed_; ++i)
      failed_ = cudaEventCreateWithFlags(&slots_[i].done, cudaEventDisableTiming) != cudaSuccess;
    if (failed_) {  // (the driver's path still works)
      cudaGetLastError();
      if (mem) cudaFreeHost(mem);
      return false;
    }
    for (int i = 0; i < kSlots; ++i) slots_[i].mem = static_cast<uint8_t*>(mem) + static_cast<size_t>(i) * kSlotBytes;
    return true;
  }

  Slot slots_[kSlots];
  int next_ = 0;
  bool failed_ = false;
};

}  // namespace
