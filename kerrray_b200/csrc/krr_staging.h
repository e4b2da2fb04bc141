// Copies between device buffers and a caller's pageable host arrays, through pinned staging memory
// and a few host threads.
//
// The driver copies pageable memory through a buffer of its own, one thread, one array after the
// other, and the pages of a freshly allocated result are faulted in by that thread as well: 4-6 GB/s
// into fresh pages, 17 GB/s into pages that a program gets back from its last result, and a wait per
// array.  Here the transfers are cut into pieces that go through a ring of pinned slots at the bus's
// rate (50 GB/s), while worker threads, one per 2 MB, move the pieces between the slots and the arrays
// (and take the page faults in parallel), and one wait serves all arrays.  Medians end to end with the
// driver's copies and with these, rtol 1e-6, results kept by the caller (fresh pages) and dropped:
//   fast64  128^2 (2 MB)   1.95 -> 1.30 ms   1.09 -> 0.96     256^2 (8 MB)   4.70 -> 2.17   1.82 -> 1.75
//           300^2 (11 MB)  6.20 -> 2.56      2.25 -> 1.99     400^2 (20 MB)  10.2 -> 3.55   3.5  -> 3.17
//   2.9M photons with a pageable Y0 (189 MB in, 377 MB out) 126 -> 49 ms (trace 41).
// Fewer threads below 16 MB (one per 8 MB) vary less from call to call and are up to a tenth faster into
// reused pages, but up to half slower into fresh ones (256^2 2.85, 300^2 3.55 ms); six threads at most
// instead of twelve take 13.1 ms instead of 11.6 for a 1000^2 image.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <cstring>
#include <memory>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

namespace krr_host {

// Whether the driver can copy to or from this host array directly (pinned or registered memory).
inline bool host_pinned(const void* p) {
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type != cudaMemoryTypeUnregistered;
}

struct CopySpan {
  void* dst;
  const void* src;
  size_t bytes;
};

// Owned by a device context and used under its lock: at most kSlots x kSlotBytes of pinned memory,
// allocated in groups as transfers first need them and kept for the next ones.  Where pinned memory
// cannot be had, the transfers use the slots there are, and without any the driver's pageable copies.
class Staging {
 public:
  static constexpr size_t kSlotBytes = (size_t)1 << 20;
  static constexpr int kSlots = 32, kGroup = 4;
  static constexpr size_t kBytesPerThread = (size_t)1 << 21;  // a thread more per 2 MB, up to kThreads
  static constexpr int kThreads = 12;

  // Device to host arrays, after what `s` holds now; returns when every byte is in place.
  cudaError_t out(int device, const std::vector<CopySpan>& spans, cudaStream_t s) {
    return run(device, spans, s, true, nullptr);
  }
  // Host arrays (of doubles) to the device on `s`; returns when the host arrays have been read, once,
  // and every copy is queued.  *bad (nullable) is set where a value that was read is not finite.
  cudaError_t in(int device, const std::vector<CopySpan>& spans, cudaStream_t s, std::atomic<bool>* bad) {
    return run(device, spans, s, false, bad);
  }

 private:
  char* slot_[kSlots] = {};
  cudaEvent_t ev_[kSlots] = {};
  int have_ = 0;

  // Slots for n pieces, or as many as there is pinned memory for (perhaps none).
  void ensure(int n) {
    while (have_ < std::min(n, kSlots)) {
      char* p = nullptr;
      if (cudaHostAlloc(reinterpret_cast<void**>(&p), kGroup * kSlotBytes, cudaHostAllocDefault) != cudaSuccess) {
        cudaGetLastError();
        return;
      }
      for (int k = 0; k < kGroup; ++k) {
        if (cudaEventCreateWithFlags(&ev_[have_ + k], cudaEventDisableTiming) != cudaSuccess) {
          cudaGetLastError();
          for (int j = 0; j < k; ++j) cudaEventDestroy(ev_[have_ + j]);
          cudaFreeHost(p);
          return;
        }
        slot_[have_ + k] = p + (size_t)k * kSlotBytes;
      }
      have_ += kGroup;
    }
  }

  // Without any slot: the driver's own copies of pageable memory.  What is checked goes through memory
  // of this call's own, so that the values copied are the ones checked.
  static cudaError_t copy_plain(const std::vector<CopySpan>& spans, cudaStream_t s, bool out, std::atomic<bool>* bad) {
    std::unique_ptr<char[]> own(bad ? new (std::nothrow) char[kSlotBytes] : nullptr);
    if (bad && !own) return cudaErrorMemoryAllocation;
    for (const CopySpan& x : spans) {
      const size_t step = bad ? kSlotBytes : x.bytes;
      for (size_t o = 0; o < x.bytes; o += step) {
        const size_t n = std::min(step, x.bytes - o);
        const char* src = static_cast<const char*>(x.src) + o;
        if (bad) {
          std::memcpy(own.get(), src, n);
          if (!finite_doubles(own.get(), n)) bad->store(true);
          src = own.get();
        }
        cudaError_t e = cudaMemcpyAsync(static_cast<char*>(x.dst) + o, src, n,
                                        out ? cudaMemcpyDeviceToHost : cudaMemcpyHostToDevice, s);
        if (e == cudaSuccess && bad) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) return e;
      }
    }
    return cudaStreamSynchronize(s);
  }

  static bool finite_doubles(const char* p, size_t bytes) {
    constexpr uint64_t kExp = 0x7ff0000000000000ull;
    uint64_t bad = 0;
    for (size_t i = 0; i + 8 <= bytes; i += 8) {
      uint64_t b;
      std::memcpy(&b, p + i, 8);
      bad |= (uint64_t)((b & kExp) == kExp);
    }
    return bad == 0;
  }

  // Piece i uses slot i mod slots.  Out: the first pieces are queued here, each worker waits for its
  // piece's copy, empties the slot and queues the piece that takes it next.  In: a worker waits for
  // the slot's previous copy, fills the slot and queues its copy.  `queued[slot]` tells the other
  // workers which piece the slot last held.
  cudaError_t run(int device, const std::vector<CopySpan>& spans, cudaStream_t s, bool out, std::atomic<bool>* bad) {
    std::vector<CopySpan> pieces;
    size_t total = 0;
    for (const CopySpan& x : spans) {
      for (size_t o = 0; o < x.bytes; o += kSlotBytes)
        pieces.push_back({static_cast<char*>(x.dst) + o, static_cast<const char*>(x.src) + o,
                          std::min(kSlotBytes, x.bytes - o)});
      total += x.bytes;
    }
    const int n = (int)pieces.size();
    if (n == 0) return out ? cudaStreamSynchronize(s) : cudaSuccess;
    ensure(n);
    if (have_ == 0) return copy_plain(spans, s, out, bad);
    const int slots = std::min(n, have_);
    std::vector<std::atomic<int>> queued(slots);
    for (auto& q : queued) q.store(-1);
    std::atomic<int> next{0}, failed{0};
    auto queue_piece = [&](int i) {
      const int k = i % slots;
      const CopySpan& x = pieces[i];
      cudaError_t r = out ? cudaMemcpyAsync(slot_[k], x.src, x.bytes, cudaMemcpyDeviceToHost, s)
                          : cudaMemcpyAsync(x.dst, slot_[k], x.bytes, cudaMemcpyHostToDevice, s);
      if (r == cudaSuccess) r = cudaEventRecord(ev_[k], s);
      if (r != cudaSuccess) {
        int none = 0;
        failed.compare_exchange_strong(none, (int)r);
      }
      queued[k].store(i, std::memory_order_release);
    };
    auto wait_slot = [&](int i) {  // until piece i has been queued in its slot and its copy is done
      const int k = i % slots;
      while (queued[k].load(std::memory_order_acquire) != i) {
        if (failed.load()) return false;
        std::this_thread::yield();
      }
      const cudaError_t r = cudaEventSynchronize(ev_[k]);
      if (r != cudaSuccess) {
        int none = 0;
        failed.compare_exchange_strong(none, (int)r);
      }
      return failed.load() == 0;
    };
    auto idle = [&](int k) {  // an earlier in() may still be reading the slot
      const cudaError_t r = cudaEventSynchronize(ev_[k]);
      if (r != cudaSuccess) {
        int none = 0;
        failed.compare_exchange_strong(none, (int)r);
      }
      return r == cudaSuccess;
    };
    auto work = [&]() {
      for (int i = next.fetch_add(1); i < n && !failed.load(); i = next.fetch_add(1)) {
        const CopySpan& x = pieces[i];
        const int k = i % slots;
        if (out) {
          if (!wait_slot(i)) return;
          std::memcpy(x.dst, slot_[k], x.bytes);
          if (i + slots < n) queue_piece(i + slots);
        } else {
          if (i >= slots ? !wait_slot(i - slots) : !idle(k)) return;
          std::memcpy(slot_[k], x.src, x.bytes);
          if (bad && !finite_doubles(slot_[k], x.bytes)) bad->store(true);
          queue_piece(i);
        }
      }
    };
    if (out)
      for (int i = 0; i < slots && idle(i); ++i) queue_piece(i);
    const int hw = (int)std::max(1u, std::thread::hardware_concurrency());
    const int threads = (int)std::min<size_t>((size_t)std::min(kThreads, hw), 1 + total / kBytesPerThread);
    // The workers of an out() sleep until the first piece has arrived: a trace of any length may run
    // ahead of the copies, and a thread that waits for an event keeps a core busy.  They watch for 0.2 ms
    // first, since waking up takes that long (camera states of 400^2 0.36 ms, 0.62 by sleeping workers).
    constexpr auto kWatch = std::chrono::microseconds(200);
    std::mutex gate;
    std::condition_variable opened;
    std::atomic<bool> open{!out};
    std::vector<std::thread> pool;
    for (int t = 1; t < threads; ++t) {
      try {
        pool.emplace_back([&] {
          const auto until = std::chrono::steady_clock::now() + kWatch;
          while (!open.load() && std::chrono::steady_clock::now() < until) std::this_thread::yield();
          {
            std::unique_lock<std::mutex> lk(gate);
            opened.wait(lk, [&] { return open.load(); });
          }
          cudaSetDevice(device);
          work();
        });
      } catch (...) {
        break;  // no more threads to be had: the others do the work
      }
    }
    if (out) {
      wait_slot(0);
      {
        std::lock_guard<std::mutex> lk(gate);
        open.store(true);
      }
      opened.notify_all();
    }
    work();
    for (auto& t : pool) t.join();
    return (cudaError_t)failed.load();
  }
};

}  // namespace krr_host
