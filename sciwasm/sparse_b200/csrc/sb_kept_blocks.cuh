// sb_kept_blocks.cuh -- freed device blocks kept for reuse (sb_malloc, sb_free).
//
// cudaMalloc and cudaFree map and unmap pages: 0.3 to several milliseconds a
// call for the arrays of a conversion, and differ from call to call.  Freed blocks are
// therefore kept, up to kKeepBytes per device (the oldest go first), and
// handed out again for the same (rounded) size.  csr_dia and csr_ell of a 44M-entry
// FP64 matrix on B200: 3.3 ms and more in all, 0.80 with the same kernels.
// Level sets with reordering of a 1M-row factor 6.9 -> 2.5 ms.
//   * A block may still be in use by work in flight on any stream when it is
//     freed.  It is handed out again only after a cudaFree since, which waits for
//     that work as the free of the block itself would have.  (A device
//     synchronisation waits too, but it invalidates a stream capture that
//     another thread has under way, or this one in relaxed mode; cudaMalloc and
//     cudaFree don't.)
//     One wait serves all blocks freed before it, so new blocks are taken while
//     little is kept (kEnoughBytes, and kEnoughSame blocks of one size), and only
//     then does an allocation wait.  (A plan of 30,000 rows takes 0.61 ms with a
//     new block and 0.26 with a kept one, from the fifth on; with 16 blocks of a
//     size, as a dearer wait had wanted it, from the 17th, and with four times
//     the memory.  Passes of conversions take as long with either.)
//     The wait is a cudaMalloc and cudaFree of 16 bytes beside a small block held
//     for good: the driver carves small blocks out of 2 MiB chunks, and the pair
//     takes 4 us on an idle B200 where a chunk is open, 1300 us where it maps and
//     unmaps one.  (Blocks under 2 MiB themselves cost the driver about as little,
//     so with the dearer wait coo_csr of 88k entries took 200 us a call against
//     190 without kept blocks.)
//   * Kept blocks are given back to the driver when an allocation of this
//     library fails, before it is tried once more; sb_mem_info counts them as
//     free.
//   * Pointers that did not come from here go to cudaFree as they are; freeing a
//     kept block again is an error, as it is for cudaFree.
//   * No lock is held while memory is allocated or freed, since a free waits for
//     the device's work: each device has its own list, and a thread that waits
//     for one device holds up nobody on another, whose next launch that work may
//     itself be waiting for.
//
// The calls of the CUDA runtime come through Api, so that the rules run on the
// host as well.  Api::Error is 0 for success, Api::out_of_memory() its value
// for a failed allocation, Api::clear() forgets the last error.
#pragma once

#include <stddef.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <list>
#include <mutex>
#include <unordered_map>
#include <utility>
#include <vector>

namespace sb {

template <class Api>
class KeptBlocks {
 public:
  using Error = typename Api::Error;
  static constexpr int kDevices = 64;
  static constexpr size_t kKeepBytes = 4ull << 30;
  static constexpr size_t kEnoughBytes = 3ull << 30;
  static constexpr size_t kEnoughSame = 4;
  static constexpr size_t kKeepBlocks = 2048;

  // A block of at least `bytes` on the current device `dev`.
  Error alloc(void** p, size_t bytes, int dev) {
    *p = nullptr;
    const size_t want = round_size(std::max<size_t>(bytes, 16));
    Device& d = devices_[dev];
    Error e{};
    if (!(*p = reuse(d, want))) {
      e = Api::malloc(p, want);
      if (e == Api::out_of_memory()) {
        Api::clear();
        give_back(dev, 0, 0);
        e = Api::malloc(p, want);
      }
      if (e != Error{}) {
        *p = nullptr;
        return e;
      }
    }
    std::lock_guard<std::mutex> lk(live_mu_);
    live_[*p] = {want, dev};
    return e;
  }

  // Keeps p, or frees what is not from here or too large; *twice is set when p
  // is kept already.  An error of the driver (of frees that make room, too, as
  // cudaFree reports earlier asynchronous errors) is returned.
  Error free(void* p, bool* twice) {
    *twice = false;
    size_t bytes = 0;
    int dev = -1;
    {
      std::lock_guard<std::mutex> lk(live_mu_);
      auto it = live_.find(p);
      if (it != live_.end()) {
        bytes = it->second.first;
        dev = it->second.second;
        live_.erase(it);
      }
    }
    if (dev < 0) {
      for (Device& d : devices_) {
        std::lock_guard<std::mutex> lk(d.mu);
        for (const Block& b : d.kept)
          if (b.ptr == p) {
            *twice = true;
            return Error{};
          }
      }
      return Api::free(p);
    }
    if (bytes > kKeepBytes) return Api::free(p);
    Device& d = devices_[dev];
    {
      std::lock_guard<std::mutex> lk(d.mu);
      d.kept.push_back({p, bytes, ++d.clock});
      d.kept_bytes += bytes;
    }
    return give_back(dev, kKeepBytes, kKeepBlocks);
  }

  // Gives the device's blocks back to the driver, the oldest first, until at
  // most `most` bytes in `blocks` blocks are kept.  Blocks that another thread
  // is giving back are gone on return.  A block that the driver does not take
  // stays kept.
  Error give_back(int dev, size_t most, size_t blocks) {
    Device& d = devices_[dev];
    {
      // (with `most` 0 the caller wants memory, so it waits for the others)
      std::lock_guard<std::mutex> lk(d.mu);
      if (most && d.kept_bytes <= most && d.kept.size() <= blocks) return Error{};
    }
    std::lock_guard<std::mutex> giving(d.giving);
    while (true) {
      Block b;
      uint64_t before;
      {
        std::lock_guard<std::mutex> lk(d.mu);
        if (d.kept_bytes <= most && d.kept.size() <= blocks) return Error{};
        b = d.kept.front();
        d.kept.pop_front();
        d.kept_bytes -= b.bytes;
        before = d.clock;
      }
      const Error e = Api::free(b.ptr);
      std::lock_guard<std::mutex> lk(d.mu);
      if (e != Error{}) {
        Api::clear();
        d.kept.push_front(b);
        d.kept_bytes += b.bytes;
        return e;
      }
      d.waited = std::max(d.waited, before);
    }
  }

  size_t kept_bytes(int dev) {
    std::lock_guard<std::mutex> lk(devices_[dev].mu);
    return devices_[dev].kept_bytes;
  }

  // Sizes are rounded so that nearly equal requests share a block: up by at most
  // 1/64, to a multiple of 512 bytes, and by less than 2 MiB (a page).  No
  // device has 2^62 bytes, and the last sizes would round up past zero: the
  // driver refuses those as they are.
  static size_t round_size(size_t b) {
    if (b >> 62) return b;
    size_t step = 512;
    while (step < (2u << 20) && step * 128 <= b) step <<= 1;
    return (b + step - 1) / step * step;
  }

 private:
  struct Block {
    void* ptr;
    size_t bytes;
    uint64_t freed;  // the device's clock when it was freed
  };

  struct Device {
    std::mutex mu;      // of the fields below; never held over a call of Api
    std::mutex giving;  // held by the thread that gives blocks back
    std::list<Block> kept;  // oldest first
    size_t kept_bytes = 0;
    uint64_t clock = 0;
    std::atomic<void*> held{nullptr};  // keeps a chunk of the driver's open
    uint64_t waited = 0;  // blocks freed up to here are no longer in use
  };

  // The block of this very size that was freed first, if it is (or, where
  // enough is kept, after a wait) no longer in use; else null.
  void* reuse(Device& d, size_t want) {
    for (int round = 0;; ++round) {
      uint64_t before;
      {
        std::lock_guard<std::mutex> lk(d.mu);
        size_t same = 0;
        auto first = d.kept.end();
        for (auto it = d.kept.begin(); it != d.kept.end(); ++it) {
          if (it->bytes != want) continue;
          if (same++ == 0) first = it;
          if (it->freed <= d.waited) break;
        }
        if (same && first->freed <= d.waited) {
          void* p = first->ptr;
          d.kept_bytes -= first->bytes;
          d.kept.erase(first);
          return p;
        }
        if (!same || round || (d.kept_bytes < kEnoughBytes && same < kEnoughSame)) return nullptr;
        before = d.clock;
      }
      if (!wait(d)) return nullptr;
      std::lock_guard<std::mutex> lk(d.mu);
      d.waited = std::max(d.waited, before);
    }
  }

  // Waits for the work that may use blocks freed before.
  static bool wait(Device& d) {
    void* p = nullptr;
    if (!d.held) {
      if (Api::malloc(&p, 16) == Error{}) {
        void* none = nullptr;
        if (!d.held.compare_exchange_strong(none, p)) Api::free(p);
      }
    }
    if (Api::malloc(&p, 16) != Error{} || Api::free(p) != Error{}) {
      Api::clear();  // the allocation that follows reports what is wrong
      return false;
    }
    return true;
  }

  Device devices_[kDevices];
  std::mutex live_mu_;
  std::unordered_map<void*, std::pair<size_t, int>> live_;  // pointer -> (bytes, device)
};

}  // namespace sb
