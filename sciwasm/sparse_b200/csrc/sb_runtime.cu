// sb_runtime.cu -- device memory, streams and error reporting of the C ABI.
// Stands in for MatMachJS's _malloc/_free over wasm linear memory
// (src/sequential/libs/matmachjs.wat:46-48) with device memory.
#include <algorithm>
#include <list>
#include <mutex>
#include <string.h>
#include <unordered_map>

#include "sb_common.cuh"

namespace sb {

static thread_local char g_err[512] = "";

void set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
}

int cuda_status(cudaError_t e, const char* what) {
  cudaGetLastError();  // reported here, not again at the next launch
  set_error("%s: %s (%s)", what, cudaGetErrorName(e), cudaGetErrorString(e));
  if (e == cudaErrorMemoryAllocation) return SB_ENOMEM;
  if (e == cudaErrorNoDevice || e == cudaErrorInsufficientDriver) return SB_ENODEV;
  return SB_ECUDA;
}

int ensure_device() {
  int n = 0;
  cudaError_t e = cudaGetDeviceCount(&n);
  if (e != cudaSuccess || n == 0) {
    cudaGetLastError();
    set_error("no CUDA device available (%s)", e == cudaSuccess ? "count 0" : cudaGetErrorString(e));
    return SB_ENODEV;
  }
  return SB_OK;
}

int sm_count() {
  static int cache[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return 148;
  if (cache[dev] == 0) {
    int n = 0;
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    cache[dev] = n > 0 ? n : 148;
  }
  return cache[dev];
}

int* device_status_word() {
  static std::mutex mu;
  static int* words[64] = {nullptr};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return nullptr;
  std::lock_guard<std::mutex> lk(mu);
  if (!words[dev]) {
    int* p = nullptr;
    if (cudaMalloc(&p, 64) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    cudaMemset(p, 0, 64);
    words[dev] = p;
  }
  return words[dev];
}

// Stream-ordered scratch comes from the device's default memory pool.  By
// default the pool hands freed memory back to the driver at every
// synchronisation, so each call that needs scratch would map fresh pages;
// keeping up to kPoolKeep bytes of freed scratch lets later calls reuse it.
constexpr uint64_t kPoolKeep = 2ull << 30;

static void keep_pool_memory() {
  static std::mutex mu;
  static bool done[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return;
  std::lock_guard<std::mutex> lk(mu);
  if (done[dev]) return;
  cudaMemPool_t pool;
  if (cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess) {
    uint64_t keep = kPoolKeep;
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
  }
  cudaGetLastError();
  done[dev] = true;
}

// ---------------------------------------------------------------- device memory
// cudaMalloc and cudaFree map and unmap pages: 0.1 to several milliseconds for
// the arrays of a conversion, and differ from call to call.  Freed blocks are
// therefore kept, up to kKeepBytes per device (the oldest go first), and
// handed out again for the same (rounded) size.  csr_dia and csr_ell of a 44M-entry
// FP64 matrix on B200: 3.3 ms and more in all, 0.80 with the same kernels.
// Level sets with reordering of a 1M-row factor 6.9 -> 2.5 ms.
//   * A block may still be in use by work in flight on any stream when it is
//     freed.  It is handed out again only after a cudaFree since, which waits for
//     that work as the free of the block itself would have.  (A device
//     synchronisation waits too, in 3 us against 0.66 ms for a small cudaMalloc
//     and cudaFree, but it invalidates a stream capture that another thread has
//     under way, or this one in relaxed mode; cudaMalloc and cudaFree don't.)
//     One wait serves all blocks freed before it, so new blocks are taken while
//     little is kept (kEnoughBytes, and kEnoughSame blocks of one size), and only
//     then does an allocation wait.
//   * Kept blocks are given back to the driver when an allocation of this
//     library fails, before it is tried once more; sb_mem_info counts them as
//     free.
//   * Pointers that did not come from here go to cudaFree as they are; freeing a
//     kept block again is an error, as it is for cudaFree.
namespace {

constexpr size_t kKeepBytes = 4ull << 30;
constexpr size_t kEnoughBytes = 3ull << 30;
constexpr size_t kEnoughSame = 16;
constexpr size_t kKeepBlocks = 2048;

struct Block {
  void* ptr;
  size_t bytes;
  uint64_t freed;  // the pool's clock when it was freed
};

struct Pool {
  std::list<Block> kept;  // oldest first
  size_t kept_bytes = 0;
  uint64_t synced = 0;  // the clock when a wait for the device's work last ended
};

struct Memory {
  std::mutex mu;
  uint64_t clock = 0;
  Pool pools[64];
  std::unordered_map<void*, std::pair<size_t, int>> live;  // pointer -> (bytes, device)
};
// Never destroyed: objects may still be freed while the process ends.
Memory& memory() {
  static Memory* m = new Memory;
  return *m;
}

// Sizes are rounded so that nearly equal requests share a block: up by at most
// 1/64, to a multiple of 512 bytes, and by less than 2 MiB (a page).
size_t round_size(size_t b) {
  size_t step = 512;
  while (step < (2u << 20) && step * 128 <= b) step <<= 1;
  return (b + step - 1) / step * step;
}

// Waits for the work that may use the kept blocks.
bool wait_for_uses(Pool& pool, Memory& mem) {
  void* p = nullptr;
  if (cudaMalloc(&p, 16) != cudaSuccess || cudaFree(p) != cudaSuccess) {
    cudaGetLastError();  // the allocation that follows reports what is wrong
    return false;
  }
  pool.synced = ++mem.clock;
  return true;
}

// Gives the pool's blocks back to the driver, the oldest first, until at most
// `most` bytes in `blocks` blocks are kept.
void trim(Pool& pool, size_t most, size_t blocks) {
  while (pool.kept_bytes > most || pool.kept.size() > blocks) {
    cudaFree(pool.kept.front().ptr);
    pool.kept_bytes -= pool.kept.front().bytes;
    pool.kept.pop_front();
  }
}

}  // namespace

int device_alloc(void** p, size_t bytes) {
  *p = nullptr;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= 64)
    return cuda_status(e == cudaSuccess ? cudaErrorInvalidDevice : e, "cudaGetDevice");
  const size_t want = round_size(std::max<size_t>(bytes, 16));
  Memory& mem = memory();
  std::lock_guard<std::mutex> lk(mem.mu);
  Pool& pool = mem.pools[dev];
  // the block of this very size that was freed first
  size_t same = 0;
  auto first = pool.kept.end();
  for (auto it = pool.kept.begin(); it != pool.kept.end(); ++it) {
    if (it->bytes != want) continue;
    if (same++ == 0) first = it;
    if (it->freed <= pool.synced) break;
  }
  if (same && (first->freed <= pool.synced ||
               ((pool.kept_bytes >= kEnoughBytes || same >= kEnoughSame) &&
                wait_for_uses(pool, mem)))) {
    *p = first->ptr;
    pool.kept_bytes -= first->bytes;
    pool.kept.erase(first);
    mem.live[*p] = {want, dev};
    return SB_OK;
  }
  e = cudaMalloc(p, want);
  if (e == cudaErrorMemoryAllocation && pool.kept_bytes) {
    cudaGetLastError();
    trim(pool, 0, 0);
    e = cudaMalloc(p, want);
  }
  if (e != cudaSuccess) {
    *p = nullptr;
    return cuda_status(e, "cudaMalloc");
  }
  mem.live[*p] = {want, dev};
  return SB_OK;
}

int device_free(void* p) {
  if (!p) return SB_OK;
  Memory& mem = memory();
  std::lock_guard<std::mutex> lk(mem.mu);
  auto it = mem.live.find(p);
  if (it == mem.live.end()) {
    for (const Pool& pool : mem.pools)
      for (const Block& b : pool.kept)
        if (b.ptr == p) return cuda_status(cudaErrorInvalidValue, "cudaFree(ptr)");
    SB_CHECK_CUDA(cudaFree(p));
    return SB_OK;
  }
  const size_t bytes = it->second.first;
  Pool& pool = mem.pools[it->second.second];
  mem.live.erase(it);
  if (bytes > kKeepBytes) {
    SB_CHECK_CUDA(cudaFree(p));
    return SB_OK;
  }
  trim(pool, kKeepBytes - bytes, kKeepBlocks - 1);
  pool.kept.push_back({p, bytes, ++mem.clock});
  pool.kept_bytes += bytes;
  return SB_OK;
}

int scratch_alloc(void** p, size_t bytes, cudaStream_t s) {
  *p = nullptr;
  if (bytes == 0) bytes = 16;
  keep_pool_memory();
  cudaError_t e = cudaMallocAsync(p, bytes, s);
  if (e == cudaErrorMemoryAllocation) {
    // the kept blocks of sb_free go back first
    int dev = 0;
    cudaGetLastError();
    Memory& mem = memory();
    std::lock_guard<std::mutex> lk(mem.mu);
    if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64 &&
        mem.pools[dev].kept_bytes) {
      trim(mem.pools[dev], 0, 0);
      e = cudaMallocAsync(p, bytes, s);
    }
  }
  if (e != cudaSuccess) return cuda_status(e, "cudaMallocAsync(scratch)");
  return SB_OK;
}

void scratch_free(void* p, cudaStream_t s) {
  if (p) cudaFreeAsync(p, s);
}

}  // namespace sb

using namespace sb;

extern "C" {

int sb_version(void) { return 10000; }

const char* sb_last_error(void) { return g_err; }

const char* sb_status_string(int s) {
  switch (s) {
    case SB_OK: return "ok";
    case SB_EINVAL: return "invalid argument";
    case SB_ENOMEM: return "out of device memory";
    case SB_EREFUSED: return "refused by the format admission test";
    case SB_ETIMEOUT: return "bounded device wait timed out";
    case SB_ECUDA: return "CUDA error";
    case SB_ENODEV: return "no CUDA device";
    case SB_EALIGN: return "misaligned pointer";
    default: return "unknown status";
  }
}

int sb_device_count(int* count) {
  SB_REQUIRE(count, "sb_device_count: null output");
  *count = 0;
  cudaError_t e = cudaGetDeviceCount(count);
  if (e != cudaSuccess) {
    cudaGetLastError();
    *count = 0;
  }
  return SB_OK;
}

int sb_set_device(int device) {
  int r = ensure_device();
  if (r) return r;
  SB_CHECK_CUDA(cudaSetDevice(device));
  return SB_OK;
}

int sb_malloc(void** ptr, size_t bytes) {
  SB_REQUIRE(ptr, "sb_malloc: null output");
  *ptr = nullptr;
  int r = ensure_device();
  if (r) return r;
  return device_alloc(ptr, bytes);
}

int sb_free(void* ptr) { return device_free(ptr); }

int sb_host_alloc(void** ptr, size_t bytes) {
  SB_REQUIRE(ptr, "sb_host_alloc: null output");
  *ptr = nullptr;
  int r = ensure_device();
  if (r) return r;
  if (bytes == 0) bytes = 16;
  SB_CHECK_CUDA(cudaMallocHost(ptr, bytes));
  return SB_OK;
}

int sb_host_free(void* ptr) {
  if (!ptr) return SB_OK;
  SB_CHECK_CUDA(cudaFreeHost(ptr));
  return SB_OK;
}

int sb_memcpy_htod(void* dst, const void* src, size_t bytes, void* stream) {
  if (bytes == 0) return SB_OK;
  SB_REQUIRE(dst && src, "sb_memcpy_htod: null pointer");
  SB_CHECK_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, as_stream(stream)));
  return SB_OK;
}

int sb_memcpy_dtoh(void* dst, const void* src, size_t bytes, void* stream) {
  if (bytes == 0) return SB_OK;
  SB_REQUIRE(dst && src, "sb_memcpy_dtoh: null pointer");
  SB_CHECK_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, as_stream(stream)));
  return SB_OK;
}

int sb_memcpy_dtod(void* dst, const void* src, size_t bytes, void* stream) {
  if (bytes == 0) return SB_OK;
  SB_REQUIRE(dst && src, "sb_memcpy_dtod: null pointer");
  SB_CHECK_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, as_stream(stream)));
  return SB_OK;
}

int sb_memset(void* dst, int value, size_t bytes, void* stream) {
  if (bytes == 0) return SB_OK;
  SB_REQUIRE(dst, "sb_memset: null pointer");
  SB_CHECK_CUDA(cudaMemsetAsync(dst, value, bytes, as_stream(stream)));
  return SB_OK;
}

int sb_stream_create(void** stream) {
  SB_REQUIRE(stream, "sb_stream_create: null output");
  int r = ensure_device();
  if (r) return r;
  cudaStream_t s;
  SB_CHECK_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
  *stream = reinterpret_cast<void*>(s);
  return SB_OK;
}

int sb_stream_create_priority(void** stream, int priority) {
  SB_REQUIRE(stream, "sb_stream_create_priority: null output");
  int r = ensure_device();
  if (r) return r;
  int least = 0, greatest = 0;
  SB_CHECK_CUDA(cudaDeviceGetStreamPriorityRange(&least, &greatest));
  // clamp into [greatest, least] (numerically lower is more urgent)
  const int p = priority < greatest ? greatest : (priority > least ? least : priority);
  cudaStream_t s;
  SB_CHECK_CUDA(cudaStreamCreateWithPriority(&s, cudaStreamNonBlocking, p));
  *stream = reinterpret_cast<void*>(s);
  return SB_OK;
}

int sb_stream_priority_range(int* least, int* greatest) {
  SB_REQUIRE(least && greatest, "sb_stream_priority_range: null output");
  int r = ensure_device();
  if (r) return r;
  SB_CHECK_CUDA(cudaDeviceGetStreamPriorityRange(least, greatest));
  return SB_OK;
}

int sb_stream_destroy(void* stream) {
  if (!stream) return SB_OK;
  SB_CHECK_CUDA(cudaStreamDestroy(as_stream(stream)));
  return SB_OK;
}

int sb_stream_synchronize(void* stream) {
  SB_CHECK_CUDA(cudaStreamSynchronize(as_stream(stream)));
  return SB_OK;
}

int sb_event_create(void** ev) {
  SB_REQUIRE(ev, "sb_event_create: null output");
  int r = ensure_device();
  if (r) return r;
  cudaEvent_t e;
  SB_CHECK_CUDA(cudaEventCreate(&e));
  *ev = reinterpret_cast<void*>(e);
  return SB_OK;
}

int sb_event_destroy(void* ev) {
  if (!ev) return SB_OK;
  SB_CHECK_CUDA(cudaEventDestroy(reinterpret_cast<cudaEvent_t>(ev)));
  return SB_OK;
}

int sb_event_record(void* ev, void* stream) {
  SB_REQUIRE(ev, "sb_event_record: null event");
  SB_CHECK_CUDA(cudaEventRecord(reinterpret_cast<cudaEvent_t>(ev), as_stream(stream)));
  return SB_OK;
}

int sb_event_query(void* ev) {
  SB_REQUIRE(ev, "sb_event_query: null event");
  cudaError_t e = cudaEventQuery(reinterpret_cast<cudaEvent_t>(ev));
  if (e == cudaSuccess) return 1;
  if (e == cudaErrorNotReady) {
    cudaGetLastError();
    return 0;
  }
  return cuda_status(e, "cudaEventQuery");
}

int sb_event_synchronize(void* ev) {
  SB_REQUIRE(ev, "sb_event_synchronize: null event");
  SB_CHECK_CUDA(cudaEventSynchronize(reinterpret_cast<cudaEvent_t>(ev)));
  return SB_OK;
}

int sb_stream_wait_event(void* stream, void* ev) {
  SB_REQUIRE(ev, "sb_stream_wait_event: null event");
  SB_CHECK_CUDA(cudaStreamWaitEvent(as_stream(stream), reinterpret_cast<cudaEvent_t>(ev), 0));
  return SB_OK;
}

int sb_event_elapsed_ms(void* start, void* end, float* ms) {
  SB_REQUIRE(start && end && ms, "sb_event_elapsed_ms: null argument");
  SB_CHECK_CUDA(cudaEventElapsedTime(ms, reinterpret_cast<cudaEvent_t>(start),
                                     reinterpret_cast<cudaEvent_t>(end)));
  return SB_OK;
}

int sb_device_status(int* code) {
  SB_REQUIRE(code, "sb_device_status: null output");
  *code = 0;
  int r = ensure_device();
  if (r) return r;
  int* w = device_status_word();
  if (!w) return SB_OK;
  SB_CHECK_CUDA(cudaDeviceSynchronize());
  SB_CHECK_CUDA(cudaMemcpy(code, w, sizeof(int), cudaMemcpyDeviceToHost));
  SB_CHECK_CUDA(cudaMemset(w, 0, sizeof(int)));
  return SB_OK;
}

int sb_mem_info(size_t* free_bytes, size_t* total_bytes) {
  SB_REQUIRE(free_bytes && total_bytes, "sb_mem_info: null output");
  int r = ensure_device();
  if (r) return r;
  SB_CHECK_CUDA(cudaMemGetInfo(free_bytes, total_bytes));
  int dev = 0;
  Memory& mem = memory();
  std::lock_guard<std::mutex> lk(mem.mu);
  if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64)
    *free_bytes += mem.pools[dev].kept_bytes;
  return SB_OK;
}

}  // extern "C"
