// sb_spts.cu -- level-set analysis and sparse triangular solves.
//
// Analysis: CSR_create_level_sets_with_reorder
// (src/parallel/src/sparse32.js:3010-3181).  level[i] = 0 when row i holds
// exactly one entry, otherwise 1 + the maximum (starting at 0) of level[c]
// over all entries but the last, where only columns c < i contribute (the
// reference reads the still-zero level of rows it has not reached).  Rows are
// stably counting-sorted by level (permutation, its inverse `order`), and a
// reordered CSR with columns relabelled by order[] is built.  All integer
// outputs are bit-exact.  Levels are computed by one thread per row, rows
// handed out in increasing order through a warp ticket so that every row a
// thread waits for has already been claimed by a running warp (or, for rows that
// read rows shortly before them, by one cluster in a fixed order); each wait is
// bounded.
//
// Solves (one thread per row, storage order, separately rounded mul/add, so
// the results are bit-identical to the reference's row kernels):
//   SB_SPTS_LEVEL    level by level on the reordered matrix, the row kernel
//                    of src/parallel/src/sparse_opt_32.wat:11679-11757
//                    (t = 0; t += L_ij*y_j; y_i = (b_i - t)/L_ii)
//   SB_SPTS_SYNCFREE natural order with per-row ready flags, the kernel of
//                    src/parallel/src/spts_opt_32.wat:8-117
//                    (t = b_i; t -= L_ij*y_j; y_i = t/L_ii)
//   SB_SPTS_HYBRID   level order with ready flags (no per-level barrier), the
//                    row kernel's arithmetic, as the level/sync-free hybrid of
//                    src/parallel/src/sparse_opt_32.wat:12846-13445
// SB_SPTS_LEVEL and SB_SPTS_HYBRID have the same arithmetic, so the kernel is
// chosen by the factor's shape (solve_impl): one block with its values in
// shared memory (sb_spts_window.cuh), a launch per level where there are few,
// one block with a barrier per level, or ready flags over the whole GPU.
#include <algorithm>
#include <climits>
#include <cstring>
#include <type_traits>
#include <mutex>
#include <vector>

#include "sb_common.cuh"
#include "sb_prims.cuh"
#include "sb_spts_window.cuh"

struct sb_spts_plan {
  int dtype = 0;
  int N = 0;
  long long nnz = 0;
  int nlevels = 0;
  int solvable = 0;
  int device = 0;
  const int* row_ptr = nullptr;  // caller's arrays (must outlive the plan)
  const int* col = nullptr;
  const void* val = nullptr;
  int* level = nullptr;
  int* level_ptr = nullptr;
  int* perm = nullptr;
  int* order = nullptr;
  int* rrow = nullptr;
  int* rcol = nullptr;
  void* rval = nullptr;
  void* ywork = nullptr;
  int* ticket = nullptr;
  // window layout (in the memory of rcol and rval, which are then not stored)
  sb::win::Info window = {};
  int4* groups = nullptr;
  char* records = nullptr;
  std::vector<void*> owned;
  cudaEvent_t ev[2] = {nullptr, nullptr};  // bracket the analysis's device work
  float analysis_ms = 0.f;
};

namespace sb {

constexpr int kT = 256;
constexpr long long kDefaultSpin = 1LL << 31;  // SM cycles (about a second)

// Polling back-off of the dependency waits: the sleep between two polls of a
// ready flag starts at SB_SPTS_SLEEP_MIN_NS and doubles up to
// SB_SPTS_SLEEP_MAX_NS.  Measured on B200 over maxima of 64 to 2048 ns (and no
// sleep), the wake-up delay of the longer sleeps costs more per level than
// the extra polling traffic of the short ones, from 190-level to 100,000-level
// factors; 64 ns was best or within 5% of best on every matrix tried.
#ifndef SB_SPTS_SLEEP_MIN_NS
#define SB_SPTS_SLEEP_MIN_NS 32u
#endif
#ifndef SB_SPTS_SLEEP_MAX_NS
#define SB_SPTS_SLEEP_MAX_NS 64u
#endif

static unsigned grid1(long long n) {
  long long g = (n + kT - 1) / kT;
  return (unsigned)std::max(1LL, std::min(g, 0x7fffffffLL));
}

__device__ __forceinline__ unsigned ld_relaxed_u32(const unsigned* p) {
  unsigned v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ void fence_acquire() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ void st_release(unsigned* p, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// Wait until flags[c] != 0 or the clock bound passes (then record a timeout
// in the status word and carry on, so that the kernel always terminates).
// Polls with relaxed loads: the caller issues an acquire fence before it
// reads what the flag publishes.
__device__ __noinline__ void wait_ready(const unsigned* flags, int c, long long limit,
                                        int* status) {
  const long long t0 = clock64();
  unsigned ns = SB_SPTS_SLEEP_MIN_NS;
  while (!ld_relaxed_u32(flags + c)) {
    // once any wait has given up, the others give up at once
    if (clock64() - t0 > limit || *(volatile const int*)status) {
      atomicExch(status, SB_DEV_TIMEOUT_DEP);
      return;
    }
    __nanosleep(ns);
    ns = ns < SB_SPTS_SLEEP_MAX_NS ? 2 * ns : ns;
  }
}

// Rows in increasing order, 32 per warp ticket.
__device__ __forceinline__ int next_rows(int* ticket) {
  int base = 0;
  if ((threadIdx.x & 31) == 0) base = atomicAdd(ticket, 32);
  return __shfl_sync(0xffffffffu, base, 0);
}

// ------------------------------------------------------------ pending values
// The plan-based solves and the level analysis publish each row's result in a
// work array that starts filled with all-one bits ("pending").  One relaxed
// load of a dependency then gives both its readiness and its value: no ready
// flag, no fence, and the loads of a row's dependencies go out together
// (kG per round trip).  A result that happens to have the pending bits is
// stored as a canonical NaN instead, so a written result is never pending.
__device__ __forceinline__ float ld_relaxed(const float* p) {
  float v;
  asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ double ld_relaxed(const double* p) {
  double v;
  asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ int ld_relaxed(const int* p) {
  int v;
  asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ void st_relaxed(float* p, float v) {
  asm volatile("st.relaxed.gpu.global.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory");
}
__device__ __forceinline__ void st_relaxed(double* p, double v) {
  asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}
__device__ __forceinline__ void st_relaxed(int* p, int v) {
  asm volatile("st.relaxed.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ bool pending(float v) { return __float_as_uint(v) == 0xffffffffu; }
__device__ __forceinline__ bool pending(double v) { return __double_as_longlong(v) == -1LL; }
__device__ __forceinline__ bool pending(int v) { return v < 0; }
__device__ __forceinline__ float settled(float v) {
  return pending(v) ? __uint_as_float(0x7fffffffu) : v;
}
__device__ __forceinline__ double settled(double v) {
  return pending(v) ? __longlong_as_double(0x7fffffffffffffffLL) : v;
}

constexpr int kG = 8;  // dependencies loaded per round trip

// Wait until none of v[k] (k < n, loaded from p[c[k]]) is pending: every
// poll reloads all still-pending entries of the group at once (one round
// trip).  The sleep between polls backs off; past the clock bound (or once
// any other wait has given up) the wait records a timeout in the status
// word and returns with the entries still pending, so that the kernel
// always terminates.
template <typename V>
__device__ __forceinline__ void wait_group(const V* p, const int (&c)[kG], V (&v)[kG], int n,
                                           long long limit, int* status) {
  unsigned mask = 0;
#pragma unroll
  for (int k = 0; k < kG; ++k)
    if (k < n && pending(v[k])) mask |= 1u << k;
  if (!mask) return;
  const long long t0 = clock64();
  unsigned ns = SB_SPTS_SLEEP_MIN_NS;
  while (true) {
    __nanosleep(ns);
    ns = ns < SB_SPTS_SLEEP_MAX_NS ? 2 * ns : ns;
#pragma unroll
    for (int k = 0; k < kG; ++k)
      if (mask & (1u << k)) v[k] = ld_relaxed(p + c[k]);
    unsigned still = 0;
#pragma unroll
    for (int k = 0; k < kG; ++k)
      if ((mask & (1u << k)) && pending(v[k])) still |= 1u << k;
    mask = still;
    if (!mask) return;
    if (clock64() - t0 > limit || *(volatile const int*)status) {
      atomicExch(status, SB_DEV_TIMEOUT_DEP);
      return;
    }
  }
}

// acc (+|-)= val[j] * w[col[j]] for j in [s, e), in storage order, waiting
// for each w[col[j]] to be published (SUB selects the sync-free form).
template <typename T, typename A, bool SUB>
__device__ __forceinline__ A dot_published(const int* __restrict__ col, const T* __restrict__ val,
                                           int s, int e, const T* w, A acc, long long limit,
                                           int* status) {
  for (int j0 = s; j0 < e; j0 += kG) {
    const int n = e - j0 < kG ? e - j0 : kG;
    int c[kG];
    A a[kG];
    T v[kG];
#pragma unroll
    for (int k = 0; k < kG; ++k)
      if (k < n) {
        c[k] = col[j0 + k];
        a[k] = (A)val[j0 + k];
      }
#pragma unroll
    for (int k = 0; k < kG; ++k)
      if (k < n) v[k] = ld_relaxed(w + c[k]);
    wait_group(w, c, v, n, limit, status);
#pragma unroll
    for (int k = 0; k < kG; ++k)
      if (k < n) acc = SUB ? sub_rn(acc, mul_rn(a[k], (A)v[k])) : add_rn(acc, mul_rn(a[k], (A)v[k]));
  }
  return acc;
}

// ------------------------------------------------------------ analysis

// What one pass over the structure tells: lower_bad = 1 unless every row is
// non-empty, ends with its diagonal and has all other columns in [0, i) (the
// structure the solves require); and how many rows read a row less than
// kNearRows before them, and one less than kClusterRows before them.
constexpr int kNearRows = 32;       // the rows of a warp
constexpr int kClusterBlocks = 8;   // the largest portable cluster
constexpr int kClusterThreads = 256;
constexpr int kClusterRows = kClusterBlocks * kClusterThreads;

struct Shape {
  int lower_bad;
  int top;          // the highest level
  int near_rows;    // rows with a dependency in the kNearRows before
  int reach_rows;   // rows with one in the kClusterRows before
  int ticket;       // rows handed out
  int status;       // a wait's timeout
};

__global__ void shape_check(const int* __restrict__ row_ptr, const int* __restrict__ col, int N,
                            Shape* __restrict__ shape) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  bool ok = true;
  int last = -1;  // the nearest row before i that it reads
  if (i < N) {
    const int s = row_ptr[i], e = row_ptr[i + 1];
    ok = e > s && col[e - 1] == i;
    for (int j = s; j < e - 1; ++j) {
      const int c = col[j];
      ok = ok && c >= 0 && c < i;
      if (c < i) last = max(last, c);
    }
  }
  const int near = __syncthreads_count(last >= 0 && i - last < kNearRows);
  const int reach = __syncthreads_count(last >= 0 && i - last < kClusterRows);
  const int bad = __syncthreads_or(!ok);
  if (threadIdx.x == 0) {
    if (near) atomicAdd(&shape->near_rows, near);
    if (reach) atomicAdd(&shape->reach_rows, reach);
    if (bad) shape->lower_bad = 1;
  }
}

// Columns of up to kG entries from s on of row i, but its last (-1: none, or
// outside [0, i), which reads as level 0).
__device__ __forceinline__ void row_columns(const int* __restrict__ col, int i, int s, int e,
                                            int (&c)[kG]) {
#pragma unroll
  for (int k = 0; k < kG; ++k) {
    const int cc = s + k < e - 1 ? __ldg(col + s + k) : -1;
    c[k] = cc < i ? cc : -1;
  }
}

// Entries of a lane's row that name rows of its own warp (rows base ..
// base + 31, one per lane) take their levels from registers: chains inside a
// warp (a stencil in natural order reads row i - 1) cost a shuffle a row
// instead of a trip through L2.  lv: a lane's level, -1 until known; inner: the
// entries waited for.
__device__ __forceinline__ void take_inner(const int (&c)[kG], int base, int lv, unsigned& inner,
                                           int& m) {
  const unsigned any = __reduce_or_sync(0xffffffffu, inner);
#pragma unroll
  for (int k = 0; k < kG; ++k)
    if (any & (1u << k)) {
      const int v = __shfl_sync(0xffffffffu, lv, c[k] - base);
      if ((inner & (1u << k)) && v >= 0) {
        m = max(m, v);
        inner &= ~(1u << k);
      }
    }
}

// One warp per 32 rows, in order (tickets).  Before the chains inside a warp
// went through registers, 3-D Laplacians took 0.56 / 2.2 / 4.9 ms (64^3 /
// 100^3 / 128^3, analysis in all, on B200), now 0.37 / 1.06 / 2.2, 100k rows
// with band 50 18.1, now 8.6.  More than `few` blocks (two per SM) pay where
// such chains hold rows back (0.43 -> 0.37 ms on 64^3) and cost where rows only
// wait for far ones (300k rows, band 100k: 0.41 -> 0.63 ms), so the others leave
// unless half the rows read one of the kNearRows before them.
__global__ void level_kernel(const int* __restrict__ row_ptr, const int* __restrict__ col, int N,
                             int* level, Shape* __restrict__ shape, int few, long long limit) {
  if ((int)blockIdx.x >= few && 2LL * shape->near_rows < N) return;
  const int lane = threadIdx.x & 31;
  int top = 0;
  while (true) {
    const int base = next_rows(&shape->ticket);
    if (base >= N) break;
    const int i = base + lane;
    int s = 0, e = 1, j0 = 0, m = 0, lv = i < N ? -1 : 0, spins = 0;
    int c[kG];
    unsigned outer = 0, inner = 0;
    if (i < N) {
      j0 = s = row_ptr[i];
      e = row_ptr[i + 1];
    }
    row_columns(col, i, s, e, c);
#pragma unroll
    for (int k = 0; k < kG; ++k)
      if (c[k] >= base) inner |= 1u << k;
      else if (c[k] >= 0) outer |= 1u << k;
    unsigned ns = SB_SPTS_SLEEP_MIN_NS;
    long long t0 = 0;
    while (true) {
      if (outer) {
        int v[kG];
#pragma unroll
        for (int k = 0; k < kG; ++k)
          if (outer & (1u << k)) v[k] = ld_relaxed(level + c[k]);
#pragma unroll
        for (int k = 0; k < kG; ++k)
          if ((outer & (1u << k)) && v[k] >= 0) {
            m = max(m, v[k]);
            outer &= ~(1u << k);
          }
      }
      bool known;
      do {
        known = false;
        if (lv < 0 && !(outer | inner)) {
          j0 += kG;
          if (j0 < e - 1) {  // a long row's next entries
            row_columns(col, i, j0, e, c);
#pragma unroll
            for (int k = 0; k < kG; ++k)
              if (c[k] >= base) inner |= 1u << k;
              else if (c[k] >= 0) outer |= 1u << k;
            known = inner != 0;  // take what is known already
          } else {
            lv = e - s == 1 ? 0 : 1 + m;
            st_relaxed(level + i, lv);
            known = true;
          }
        }
        known = __any_sync(0xffffffffu, known);
        if (known) take_inner(c, base, lv, inner, m);
      } while (known);
      if (!__any_sync(0xffffffffu, lv < 0)) break;
      if (++spins > 1) {
        __nanosleep(ns);
        ns = ns < SB_SPTS_SLEEP_MAX_NS ? 2 * ns : ns;
        if ((spins & 255) == 0) {
          if (t0 == 0) t0 = clock64();
          if (clock64() - t0 > limit || *(volatile const int*)&shape->status) {
            // the call fails; the rows that waited end at a level of their own
            atomicExch(&shape->status, SB_DEV_TIMEOUT_DEP);
            if (lv < 0) st_relaxed(level + i, lv = 0);
            outer = inner = 0;
          }
        }
      }
    }
    top = max(top, lv);
  }
  top = __reduce_max_sync(0xffffffffu, top);
  if (lane == 0 && top > 0) atomicMax(&shape->top, top);
}

// The same on one cluster of kClusterBlocks blocks, for factors whose rows
// mostly read rows a little before them: each block keeps the levels of the
// last kRing rows in its shared memory, and a row's level is stored into every
// block's ring, so a dependency costs a store across the cluster and a
// shared-memory poll (0.55 us) rather than two trips through L2 (1.3 us).
// A ring entry is one 64-bit word, the row (plus 1) above its level, so a
// reader can tell its row's entry from an older one (poll on) or a newer one
// (the entry is gone: read the level's global word, -1 until it is there).
// Stores of different blocks to one slot may land in either order, which could
// leave an older row's entry for good, so a long wait turns to global memory
// as well; no wait depends on the ring alone.  Consecutive 32-row chunks go to
// different blocks; the lowest unfinished row always has its warp running and
// its dependencies published, and a row publishes its level while others of
// its warp still wait.
//
// It runs where at least 3/4 of the rows read one of the kClusterRows before
// them (those in flight: with fewer, rows far apart are independent and the
// whole GPU is the better place) and less than half read one of the kNearRows
// before them (chains inside a warp: a stencil in natural order); otherwise it
// leaves the ticket at 0 and level_kernel takes all rows.  Analysis in all,
// level_kernel alone -> with this one, on B200: 1M-row random factor with band
// 5000 4.7 -> 2.3 ms, 100k rows with band 500 2.3 -> 1.9; without the rule a 3-D
// Laplacian 64^3 would take 2.3 instead of 0.4, 300k rows with band 100k 0.73
// instead of 0.41.  Fewer or more blocks or warps, sleeping between polls, rows
// spread over the warps and one block sweeping over 1024 rows at a time were
// slower.
constexpr int kRing = 16384;  // entries: 128 KB

__device__ __forceinline__ unsigned long long ld_entry(uint32_t a) {
  unsigned long long v;
  asm volatile("ld.relaxed.cluster.shared::cta.u64 %0, [%1];" : "=l"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void st_entry(uint32_t a, unsigned long long v) {
  asm volatile("st.relaxed.cluster.shared::cluster.u64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
}
__device__ __forceinline__ uint32_t peer_address(uint32_t a, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_barrier() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::
                   : "memory");
}

// Which of a row's entries lie in the ring, and which are too far back for it.
__device__ __forceinline__ void row_waits(const int (&c)[kG], int i, unsigned& pend,
                                          unsigned& far) {
#pragma unroll
  for (int k = 0; k < kG; ++k)
    if (c[k] >= 0) {
      if (i - c[k] < kRing) pend |= 1u << k;
      else far |= 1u << k;
    }
}

__global__ void __launch_bounds__(kClusterThreads, 1)
    level_cluster_kernel(const int* __restrict__ row_ptr, const int* __restrict__ col, int N,
                         int* level, Shape* __restrict__ shape, long long limit) {
  extern __shared__ __align__(16) unsigned long long ring[];
  int* status = &shape->status;
  int top = 0;
  if (4LL * shape->reach_rows < 3LL * N || 2LL * shape->near_rows >= N) return;
  for (int k = threadIdx.x; k < kRing; k += kClusterThreads) ring[k] = 0;
  const uint32_t own = smem_u32(ring);
  uint32_t peer[kClusterBlocks];
#pragma unroll
  for (int r = 0; r < kClusterBlocks; ++r) peer[r] = peer_address(own, r);
  cluster_barrier();
  const int lane = threadIdx.x & 31;
  constexpr int step = kClusterRows;
  int i = 32 * ((threadIdx.x >> 5) * kClusterBlocks + (int)blockIdx.x) + lane;
  int s = 0, e = 0, s1 = 0, e1 = 0;
  int c[kG], c1[kG];
#pragma unroll
  for (int k = 0; k < kG; ++k) c[k] = c1[k] = -1;
  if (i < N) {
    s = __ldg(row_ptr + i);
    e = __ldg(row_ptr + i + 1);
    row_columns(col, i, s, e, c);
  }
  if (i + (long long)step < N) {
    s1 = __ldg(row_ptr + i + step);
    e1 = __ldg(row_ptr + i + step + 1);
  }
  for (long long first = i - lane; first < N; first += step) {
    // ahead: the next row's columns and the bounds of the row after it
    const bool next = i + (long long)step < N, second = i + 2LL * step < N;
    if (next) row_columns(col, i + step, s1, e1, c1);
    int s2 = 0, e2 = 0;
    if (second) {
      s2 = __ldg(row_ptr + i + 2 * step);
      e2 = __ldg(row_ptr + i + 2 * step + 1);
    }
    bool waiting = first + lane < N;
    int m = 0, j0 = s, spins = 0;
    unsigned pend = 0, far = 0;
    row_waits(c, i, pend, far);
    long long t0 = 0;
    while (__any_sync(0xffffffffu, waiting)) {
      if (waiting) {
        unsigned long long w[kG];
#pragma unroll
        for (int k = 0; k < kG; ++k)
          if (pend & (1u << k)) w[k] = ld_entry(own + (uint32_t)(c[k] & (kRing - 1)) * 8u);
#pragma unroll
        for (int k = 0; k < kG; ++k)
          if (pend & (1u << k)) {
            const int ahead = (int)(w[k] >> 32) - (c[k] + 1);
            if (ahead == 0) m = max(m, (int)w[k]);
            if (ahead >= 0) pend &= ~(1u << k);
            if (ahead > 0) far |= 1u << k;
          }
        const bool long_wait = (++spins & 63) == 0;
        if (far || long_wait) {
          const unsigned ask = far | (long_wait ? pend : 0u);
#pragma unroll
          for (int k = 0; k < kG; ++k)
            if (ask & (1u << k)) {
              const int v = ld_relaxed(level + c[k]);
              if (v >= 0) {
                m = max(m, v);
                far &= ~(1u << k);
                pend &= ~(1u << k);
              }
            }
        }
        if (!(pend | far)) {
          j0 += kG;
          if (j0 < e - 1) {  // a long row's next entries
            row_columns(col, i, j0, e, c);
            row_waits(c, i, pend, far);
          } else {
            const int lv = e - s == 1 ? 0 : 1 + m;
            const unsigned long long v =
                (unsigned long long)(unsigned)(i + 1) << 32 | (unsigned)lv;
            const uint32_t o = (uint32_t)(i & (kRing - 1)) * 8u;
#pragma unroll
            for (int r = 0; r < kClusterBlocks; ++r) st_entry(peer[r] + o, v);
            st_relaxed(level + i, lv);
            top = max(top, lv);
            waiting = false;
          }
        } else if ((spins & 1023) == 0) {
          if (t0 == 0) t0 = clock64();
          if (clock64() - t0 > limit || *(volatile const int*)status) {
            atomicExch(status, SB_DEV_TIMEOUT_DEP);
            st_relaxed(level + i, 0);  // the call fails; the kernel ends
            waiting = false;
          }
        }
      }
    }
    s = s1;
    e = e1;
    s1 = s2;
    e1 = e2;
    i = next ? i + step : i;
#pragma unroll
    for (int k = 0; k < kG; ++k) c[k] = next ? c1[k] : -1;
  }
  top = __reduce_max_sync(0xffffffffu, top);
  if (lane == 0 && top > 0) atomicMax(&shape->top, top);
  cluster_barrier();  // no block leaves while others still store into its ring
  if (blockIdx.x == 0 && threadIdx.x == 0) shape->ticket = N;
}

__global__ void level_hist(const int* __restrict__ level, int N, int* __restrict__ counts) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < N) atomicAdd(counts + level[i], 1);
}

__global__ void level_keys(const int* __restrict__ level, int N, unsigned long long* __restrict__ k,
                           unsigned* __restrict__ v) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < N) {
    k[i] = (unsigned long long)(unsigned)level[i];
    v[i] = (unsigned)i;
  }
}

__global__ void perm_order(const unsigned* __restrict__ sorted_rows, int N, int* __restrict__ perm,
                           int* __restrict__ order) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < N) {
    const int i = (int)sorted_rows[p];
    perm[p] = i;
    order[i] = p;
  }
}

// Not run where the window layout takes the memory (info->use).
template <typename T>
__global__ void reorder_rows(const int* __restrict__ row_ptr, const int* __restrict__ col,
                             const T* __restrict__ val, const int* __restrict__ perm,
                             const int* __restrict__ order, const int* __restrict__ rrow, int N,
                             const win::Info* __restrict__ info, int* __restrict__ rcol,
                             T* __restrict__ rval) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= N || info->use) return;
  const int src = perm[p];
  int o = rrow[p];
  for (int j = row_ptr[src]; j < row_ptr[src + 1]; ++j, ++o) {
    const int c = col[j];
    rcol[o] = (c >= 0 && c < N) ? order[c] : c;
    rval[o] = val[j];
  }
}

// ------------------------------------------------------------ solves

// One level of few: a launch each, a thread per row, with nothing to wait for
// and no pending values to fill in.  Up to kFewLevels the launches cost less than
// the ready flags, or a grid barrier per level (the whole call of 1M FP64 rows on
// B200, flags / grid barriers / so: 1 level 55 / 43 / 32 us, 3 levels 65 / 56 / 42).
constexpr int kFewLevels = 4;

template <typename T, typename A>
__global__ void spts_level_rows(const int* __restrict__ rrow, const int* __restrict__ rcol,
                                const T* __restrict__ rval, const int* __restrict__ level_ptr,
                                int l, const int* __restrict__ perm, const T* __restrict__ b,
                                T* yw, T* __restrict__ y) {
  const int i = level_ptr[l] + (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (i >= level_ptr[l + 1]) return;
  const int s = rrow[i], end = rrow[i + 1] - 1, pi = perm[i];
  const A bi = (A)b[pi];
  T yi;
  if (end > s) {
    A t = 0;
    for (int j = s; j < end; ++j) t = add_rn(t, mul_rn((A)rval[j], (A)yw[rcol[j]]));
    yi = (T)div_rn(sub_rn(bi, t), (A)rval[end]);
  } else {
    yi = (T)div_rn(bi, (A)rval[end]);
  }
  yw[i] = yi;
  y[pi] = yi;
}

// A thread's first row of a level, read ahead of the barrier that opens the
// level: its structure, b, diagonal and up to kG off-diagonal columns and
// values (the values of the columns are read after the barrier).
template <typename T, typename A>
struct LevelRow {
  int i = -1, s = 0, end = 0, pi = 0;
  A bi = 0, diag = 0;
  int c[kG];
  A v[kG];
};

// A thread's first row of the level after next: where its entries are and
// where its output goes (the first of the two dependent load rounds of a
// row, issued one level earlier than the second).
struct LevelHead {
  int i = -1, s = 0, end = 0, pi = 0;
};

__device__ __forceinline__ void level_head_load(LevelHead& h, int i, const int* rrow,
                                                const int* perm) {
  h.i = i;
  h.s = rrow[i];
  h.end = rrow[i + 1] - 1;
  h.pi = perm[i];
}

// The second round: b, the diagonal and up to kG off-diagonal columns and
// values of the row a head describes.
template <typename T, typename A>
__device__ __forceinline__ void level_row_from_head(LevelRow<T, A>& r, const LevelHead& h,
                                                    const int* rcol, const T* rval, const T* b) {
  r.i = h.i;
  if (h.i < 0) return;
  r.s = h.s;
  r.end = h.end;
  r.pi = h.pi;
  r.bi = (A)b[r.pi];
  r.diag = (A)rval[r.end];
#pragma unroll
  for (int k = 0; k < kG; ++k) {
    const int j = r.s + k;
    r.c[k] = j < r.end ? rcol[j] : 0;
    r.v[k] = j < r.end ? (A)rval[j] : A(0);
  }
}

template <typename T, typename A>
__device__ __forceinline__ void level_row_load(LevelRow<T, A>& r, int i, const int* rrow,
                                               const int* rcol, const T* rval, const int* perm,
                                               const T* b) {
  r.i = i;
  r.s = rrow[i];
  r.end = rrow[i + 1] - 1;
  r.pi = perm[i];
  r.bi = (A)b[r.pi];
  r.diag = (A)rval[r.end];
#pragma unroll
  for (int k = 0; k < kG; ++k) {
    const int j = r.s + k;
    r.c[k] = j < r.end ? rcol[j] : 0;
    r.v[k] = j < r.end ? (A)rval[j] : A(0);
  }
}

// The level-set solve of a factor whose levels all fit one block of
// kLevelBlock threads: the levels in order, one row per thread, a block barrier
// after every level (the reference's structure,
// src/parallel/src/spts_opt_32.wat:339-546).  Values of earlier levels are
// read from L2 (__ldcg); each row also writes its natural-order output, so no
// scatter pass follows.  Each thread reads its row of a level ahead of time
// (TWO: in two rounds, its row pointers and permutation two levels before, its
// columns, values, b and diagonal one level before), so that only the y reads
// after each barrier lie on the level's critical path.  Wider levels go to the
// ready flags of spts_hybrid_rows: a grid barrier per level measured 2.1 us
// per level against their 1.3 (3-D Laplacian 64^3 FP64, 0.41 and 0.25 ms).
constexpr int kLevelBlock = 512;

template <typename T, typename A, bool TWO>
__global__ void __launch_bounds__(kLevelBlock, 1)
    spts_level_block(const int* __restrict__ rrow, const int* __restrict__ rcol,
                     const T* __restrict__ rval, const int* __restrict__ level_ptr, int nlevels,
                     const int* __restrict__ perm, const T* __restrict__ b, T* yw,
                     T* __restrict__ y) {
  const int gt = threadIdx.x;
  LevelRow<T, A> nx;
  LevelHead hd;  // the row of the level after the next one
  {
    const int r0 = __ldg(level_ptr), r1 = __ldg(level_ptr + 1);
    if (r0 + gt < r1) level_row_load(nx, r0 + gt, rrow, rcol, rval, perm, b);
    if (TWO && nlevels > 1) {
      const int q0 = r1, q1 = __ldg(level_ptr + 2);
      if (q0 + gt < q1) level_head_load(hd, q0 + gt, rrow, perm);
    }
  }
  for (int l = 0; l < nlevels; ++l) {
    const int r1 = __ldg(level_ptr + l + 1);
    if (nx.i >= 0) {
      A t = 0;
      const int n = nx.end - nx.s;
      T w[kG];
#pragma unroll
      for (int k = 0; k < kG; ++k)
        if (k < n) w[k] = __ldcg(yw + nx.c[k]);
#pragma unroll
      for (int k = 0; k < kG; ++k)
        if (k < n) t = add_rn(t, mul_rn(nx.v[k], (A)w[k]));
      for (int j = nx.s + kG; j < nx.end; ++j)
        t = add_rn(t, mul_rn((A)rval[j], (A)__ldcg(yw + rcol[j])));
      const T yi = n > 0 ? (T)div_rn(sub_rn(nx.bi, t), nx.diag) : (T)div_rn(nx.bi, nx.diag);
      __stcg(yw + nx.i, yi);
      y[nx.pi] = yi;
    }
    if (l + 1 < nlevels) {
      if constexpr (TWO) {
        // the next level's row from the head read one level ago, and the head
        // of the level after it: neither depends on y, so both load rounds
        // overlap the barrier and the next level's y reads
        level_row_from_head(nx, hd, rcol, rval, b);
        hd.i = -1;
        if (l + 2 < nlevels) {
          const int q0 = __ldg(level_ptr + l + 2), q1 = __ldg(level_ptr + l + 3);
          if (q0 + gt < q1) level_head_load(hd, q0 + gt, rrow, perm);
        }
      } else {
        // both rounds of the next level's row, before the barrier
        const int q1 = __ldg(level_ptr + l + 2);
        nx.i = -1;
        if (r1 + gt < q1) level_row_load(nx, r1 + gt, rrow, rcol, rval, perm, b);
      }
      __syncthreads();  // orders the block's L2 accesses
    }
  }
}

// Level-ordered rows (hybrid): same arithmetic as above, dependencies read
// from the pending-initialised work vector yw (level order); each row also
// writes its natural-order output y[perm[i]].
template <typename T, typename A>
__global__ void spts_hybrid_rows(const int* __restrict__ rrow, const int* __restrict__ rcol,
                                 const T* __restrict__ rval, int N, const int* __restrict__ perm,
                                 const T* __restrict__ b, T* yw, T* __restrict__ y,
                                 int* __restrict__ ticket, long long limit, int* status) {
  while (true) {
    const int base = next_rows(ticket) + 1;  // (-1 at first, as all pending words)
    if (base >= N) return;
    const int i = base + (threadIdx.x & 31);
    if (i < N) {
      const int s = rrow[i], end = rrow[i + 1] - 1;
      const int pi = perm[i];
      const A bi = (A)b[pi];
      T yi;
      if (end > s) {
        const A t = dot_published<T, A, false>(rcol, rval, s, end, yw, A(0), limit, status);
        yi = (T)div_rn(sub_rn(bi, t), (A)rval[end]);
      } else {
        yi = (T)div_rn(bi, (A)rval[end]);
      }
      st_relaxed(yw + i, settled(yi));
      y[pi] = yi;
    }
  }
}

// Sync-free solve of an analysed (lower, diagonal last) matrix in natural
// order, the sync-free kernel's arithmetic (t = b_i; t -= L_ij*y_j;
// y_i = t/L_ii), dependencies read from the pending-initialised yw.
template <typename T, typename A>
__global__ void spts_syncfree_plan_rows(const int* __restrict__ row_ptr,
                                        const int* __restrict__ col, const T* __restrict__ val,
                                        int N, const T* __restrict__ b, T* yw, T* __restrict__ y,
                                        int* __restrict__ ticket, long long limit, int* status) {
  while (true) {
    const int base = next_rows(ticket) + 1;  // (-1 at first, as all pending words)
    if (base >= N) return;
    const int i = base + (threadIdx.x & 31);
    if (i < N) {
      const int s = row_ptr[i], e = row_ptr[i + 1];
      const A t = dot_published<T, A, true>(col, val, s, e - 1, yw, (A)b[i], limit, status);
      const T yi = (T)div_rn(t, (A)val[e - 1]);
      st_relaxed(yw + i, settled(yi));
      y[i] = yi;
    }
  }
}

// Sync-free solve in natural order (t = b_i; t -= L_ij*y_j; y_i = t/L_ii) on
// the caller's arrays with ready flags: a row first waits for the flags of
// all its in-range dependencies (kG relaxed loads per round trip), then one
// acquire fence orders the value loads after them.
template <typename T, typename A>
__global__ void spts_syncfree_rows(const int* __restrict__ row_ptr, const int* __restrict__ col,
                                   const T* __restrict__ val, int N, const T* __restrict__ b, T* y,
                                   unsigned* __restrict__ done, int* __restrict__ ticket,
                                   long long limit, int* status) {
  while (true) {
    const int base = next_rows(ticket);
    if (base >= N) return;
    const int i = base + (threadIdx.x & 31);
    if (i < N) {
      const int s = row_ptr[i], e = row_ptr[i + 1];
      A t = (A)b[i];
      T yi;
      if (e > s + 1) {
        for (int j0 = s; j0 < e - 1; j0 += kG) {
          int c[kG];
          unsigned f[kG];
#pragma unroll
          for (int k = 0; k < kG; ++k) c[k] = (j0 + k < e - 1) ? col[j0 + k] : -1;
#pragma unroll
          for (int k = 0; k < kG; ++k) f[k] = (c[k] >= 0 && c[k] < N) ? ld_relaxed_u32(done + c[k]) : 1u;
#pragma unroll
          for (int k = 0; k < kG; ++k)
            if (!f[k]) wait_ready(done, c[k], limit, status);
        }
        fence_acquire();
        for (int j0 = s; j0 < e - 1; j0 += kG) {
          int c[kG];
          T v[kG];
#pragma unroll
          for (int k = 0; k < kG; ++k) c[k] = (j0 + k < e - 1) ? col[j0 + k] : -1;
#pragma unroll
          for (int k = 0; k < kG; ++k)
            if (c[k] >= 0 && c[k] < N) v[k] = ld_relaxed(y + c[k]);
#pragma unroll
          for (int k = 0; k < kG; ++k)
            if (c[k] >= 0 && c[k] < N) t = sub_rn(t, mul_rn((A)val[j0 + k], (A)v[k]));
        }
        yi = (T)div_rn(t, (A)val[e - 1]);
      } else {
        yi = (e > s) ? (T)div_rn(t, (A)val[s]) : (T)t;
      }
      y[i] = yi;
      st_release(done + i, 1u);
    }
  }
}

// ------------------------------------------------------------ batched solves
// Plans with a window layout are solved one per block
// (win::window_solve_many); the others as follows.  Many independent systems
// in one launch of one warp per 32-row chunk (not
// persistent: warps exit after their chunk, and the hardware dispatches the
// blocks as SM slots free up).  Warps are laid out in rounds of one chunk per
// unfinished system, so all systems of a batch advance at the same time and
// the launch takes about the deepest system's time, not the sum.  A warp
// takes its chunk from its system's ticket counter, i.e. chunks of a system
// are claimed in level order by running warps; a row waits only on rows of
// its own system with a smaller level-order index, all claimed by running
// warps, so the launch always makes progress whatever order the hardware
// runs the blocks in.  Rows are solved as in spts_hybrid_rows.
constexpr int kTB = 128;  // threads per block of the batched solve

struct SptsDesc {
  const int* rrow;
  const int* rcol;
  const void* rval;
  const int* perm;
  void* yw;
  const void* b;
  void* y;
  int N;
  int pad;
};

// Schedule of one batch: systems sorted by chunk count (order[]), and the
// warps in rounds of one chunk per system still unfinished.  Segment k holds
// the rounds [nch(order[k-1]), nch(order[k])) of the M - k systems
// order[k..M-1]; seg[k] is the first warp of segment k and `warps` the
// number of warps (one per chunk of the batch).
struct SptsSched {
  int M;
  int pad;
  long long warps;
};

// Every item's work vector to the pending bits.
template <typename T>
__global__ void spts_batch_reset(const SptsDesc* __restrict__ items,
                                 const SptsSched* __restrict__ sched) {
  using U = typename std::conditional<sizeof(T) == 4, unsigned, unsigned long long>::type;
  const int M = sched->M;
  for (int k = 0; k < M; ++k) {
    U* w = (U*)items[k].yw;
    const long long N = items[k].N;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < N;
         i += (long long)gridDim.x * blockDim.x)
      w[i] = ~U(0);
  }
}

// The chunk of warp slot gw of the round layout: its system from the
// segment table, the chunk itself from the system's ticket (claimed in level
// order by a running warp), then one row per lane as in spts_hybrid_rows.
template <typename T, typename A>
__device__ __forceinline__ void batch_chunk(const SptsDesc* __restrict__ items,
                                            const int* __restrict__ order,
                                            const long long* __restrict__ seg,
                                            int* __restrict__ tickets, int M, long long gw,
                                            int lane, long long limit, int* status) {
  int lo = 0, hi = M - 1;  // last segment starting at or before gw
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (seg[mid] <= gw) lo = mid; else hi = mid - 1;
  }
  const int sys = order[lo + (int)((gw - seg[lo]) % (M - lo))];
  int t = 0;
  if (lane == 0) t = atomicAdd(tickets + sys, 1);
  t = __shfl_sync(0xffffffffu, t, 0);
  const SptsDesc d = items[sys];
  const int i = t * 32 + lane;
  if (i >= d.N) return;
  const T* __restrict__ rval = (const T*)d.rval;
  T* yw = (T*)d.yw;
  const int s = d.rrow[i], end = d.rrow[i + 1] - 1;
  const int pi = d.perm[i];
  const A bi = (A)((const T*)d.b)[pi];
  T yi;
  if (end > s) {
    const A acc = dot_published<T, A, false>(d.rcol, rval, s, end, yw, A(0), limit, status);
    yi = (T)div_rn(sub_rn(bi, acc), (A)rval[end]);
  } else {
    yi = (T)div_rn(bi, (A)rval[end]);
  }
  st_relaxed(yw + i, settled(yi));
  ((T*)d.y)[pi] = yi;
}

// persistent == 0: one warp per warp slot (the grid covers the layout).
// persistent != 0: a capped grid whose warps take warp slots from *work
// until the layout is done, so that the launch leaves SMs to other work (a
// concurrent batch on another stream).  Either way a chunk is claimed only
// by a running warp, and a row waits only on rows of its own system claimed
// earlier, so the launch always makes progress.
template <typename T, typename A>
__global__ void __launch_bounds__(kTB)
    spts_batch_kernel(const SptsDesc* __restrict__ items, const SptsSched* __restrict__ sched,
                      const int* __restrict__ order, const long long* __restrict__ seg,
                      int* __restrict__ tickets, long long limit, int* status,
                      unsigned long long* __restrict__ work, int persistent) {
  const int lane = threadIdx.x & 31;
  const int M = sched->M;
  const long long warps = sched->warps;
  if (M <= 0) return;
  if (!persistent) {
    const long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (gw < warps) batch_chunk<T, A>(items, order, seg, tickets, M, gw, lane, limit, status);
    return;
  }
  while (true) {
    unsigned long long w = 0;
    if (lane == 0) w = atomicAdd(work, 1ull);
    w = __shfl_sync(0xffffffffu, w, 0);
    if ((long long)w >= warps) return;
    batch_chunk<T, A>(items, order, seg, tickets, M, (long long)w, lane, limit, status);
    __syncwarp();
  }
}

// max over rows of sum_{j < diag} |L_ij| / |L_ii| (inf for a zero diagonal),
// as the bits of a non-negative double so that an integer max orders them.
template <typename T>
__global__ void growth_kernel(const int* __restrict__ row_ptr, const T* __restrict__ val, int N,
                              unsigned long long* __restrict__ out) {
  double m = 0.0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < N;
       i += (long long)gridDim.x * blockDim.x) {
    const int s = row_ptr[i], e = row_ptr[i + 1];
    if (e <= s) continue;
    double off = 0.0;
    for (int j = s; j < e - 1; ++j) off += fabs((double)val[j]);
    const double dg = fabs((double)val[e - 1]);
    const double r = off / dg;  // 0/0 -> NaN, x/0 -> inf
    const double rr = (r != r) ? __longlong_as_double(0x7ff0000000000000LL) : r;
    m = rr > m ? rr : m;
  }
  unsigned long long b = (unsigned long long)__double_as_longlong(m);
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long v = __shfl_xor_sync(0xffffffffu, b, o);
    b = v > b ? v : b;
  }
  if ((threadIdx.x & 31) == 0) atomicMax(out, b);
}

// flags[0] = 1 unless every column j of a CSC lower triangle is non-empty,
// starts with its diagonal (row j) and has all other rows in (j, N).
__global__ void csc_lower_check(const int* __restrict__ col_ptr, const int* __restrict__ row,
                                int N, int* __restrict__ flags) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= N) return;
  const int s = col_ptr[j], e = col_ptr[j + 1];
  bool ok = e > s && row[s] == j;
  for (int q = s + 1; ok && q < e; ++q) ok = row[q] > j && row[q] < N;
  if (!ok) flags[0] = 1;
}

static int resident_grid(const void* kern) {
  int per = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, kT, 0);
  return std::max(1, per) * sm_count();
}

// Grid of the plan-based polling solves.  Every warp that holds rows ahead
// of the dependency frontier polls, and polling warps take issue slots and
// L2 round trips from the warps at the frontier.  Measured on B200 from 74 to
// 592 CTAs, on factors with 1 to 10^6 rows per level:
//  * the level-ordered hybrid solve was fastest, or within 3%, with one CTA
//    per SM on every factor (3-D Laplacian 64^3: 0.295 -> 0.246 ms; 1M-row
//    random factor with 3470 levels: 9.5 -> 4.6 ms);
//  * the natural-order sync-free solve needs the full resident grid when
//    levels are wide (3-D Laplacians, >= 1380 rows per level: 5.6 ms at 444
//    CTAs, 9.5 ms at 148 on 128^3) and one CTA per SM when they are narrow
//    (288 rows per level: 9.5 -> 4.4 ms).
// Grid of the natural-order polling kernels that run without level
// information (the sync-free solve on caller arrays): two CTAs per SM.
// Measured on B200 against the resident grid (ms): 3-D Laplacian 64^3 1.51 ->
// 1.50; 128^3 15.2 -> 15.4; 1M-row random factor 41.0 -> 25.9; band-50 1M
// 2048 -> 1368; bidiagonal 100k 265 -> 259.  One CTA per SM was faster still on
// the narrow factors and 30-50% slower on the Laplacians.
static int natural_order_grid(const void* kern) {
  return std::min(resident_grid(kern), 2 * sm_count());
}

static int polling_grid(const void* kern, int algo, int N, int nlevels) {
  const int full = resident_grid(kern);
  const bool wide = nlevels > 0 && (long long)N >= 1024LL * nlevels;
  if (algo == SB_SPTS_SYNCFREE && wide) return full;
  return std::min(full, sm_count());
}

// The plan's device arrays live in one allocation (one per plan,
// not one per array); level_ptr is sized for the largest possible level
// count, N + 1 (a row's level is at most its index + 1).
static size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

static void plan_release(sb_spts_plan* p) {
  for (void* q : p->owned) device_free(q);
  p->owned.clear();
  if (p->ev[0]) cudaEventDestroy(p->ev[0]);
  if (p->ev[1]) cudaEventDestroy(p->ev[1]);
  p->ev[0] = p->ev[1] = nullptr;
}

static int launch_level_cluster(const sb_spts_plan* p, Shape* shape, cudaStream_t st) {
  const size_t smem = sizeof(unsigned long long) * kRing;
  SB_CHECK_CUDA(cudaFuncSetAttribute((const void*)level_cluster_kernel,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kClusterBlocks);
  cfg.blockDim = dim3(kClusterThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = kClusterBlocks;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  SB_CHECK_CUDA(cudaLaunchKernelEx(&cfg, level_cluster_kernel, p->row_ptr, p->col, p->N, p->level,
                                   shape, (long long)kDefaultSpin));
  return SB_OK;
}

template <typename T>
static int analyze_impl(sb_spts_plan* p, cudaStream_t st) {
  const int N = p->N;
  const long long nnz = p->nnz;
  int r;
  {
    const size_t sizes[9] = {sizeof(int) * (size_t)N,           sizeof(int) * (size_t)N,
                             sizeof(int) * (size_t)N,           sizeof(int) * ((size_t)N + 1),
                             sizeof(int) * (size_t)nnz,         sizeof(T) * (size_t)nnz,
                             sizeof(T) * (size_t)N,             sizeof(int) * 4,
                             sizeof(int) * ((size_t)N + 2)};
    size_t total = 0;
    for (size_t b : sizes) total += align256(b);
    void* slab = nullptr;
    if ((r = device_alloc(&slab, total))) return r;
    p->owned.push_back(slab);
    char* q = (char*)slab;
    void* part[9];
    for (int k = 0; k < 9; ++k) {
      part[k] = q;
      q += align256(sizes[k]);
    }
    p->level = (int*)part[0];
    p->perm = (int*)part[1];
    p->order = (int*)part[2];
    p->rrow = (int*)part[3];
    p->rcol = (int*)part[4];
    p->rval = part[5];
    p->ywork = part[6];
    p->ticket = (int*)part[7];
    p->level_ptr = (int*)part[8];
    SB_CHECK_CUDA(cudaEventCreate(&p->ev[0]));
    SB_CHECK_CUDA(cudaEventCreate(&p->ev[1]));
  }
  SB_CHECK_CUDA(cudaEventRecord(p->ev[0], st));
  Shape* shape = nullptr;
  if ((r = scratch_alloc((void**)&shape, sizeof(Shape), st))) return r;
  SB_CHECK_CUDA(cudaMemsetAsync(shape, 0, sizeof(Shape), st));
  shape_check<<<grid1(N), kT, 0, st>>>(p->row_ptr, p->col, N, shape);
  SB_CHECK_LAUNCH("shape_check");
  SB_CHECK_CUDA(cudaMemsetAsync(p->level, 0xff, sizeof(int) * N, st));
  // (a few thousand rows leave the cluster nothing to gain)
  if (N >= 4 * kClusterRows && (r = launch_level_cluster(p, shape, st))) return r;
  level_kernel<<<std::min(resident_grid((const void*)level_kernel), 4 * sm_count()), kT, 0, st>>>(
      p->row_ptr, p->col, N, p->level, shape, 2 * sm_count(), kDefaultSpin);
  SB_CHECK_LAUNCH("level_kernel");
  Shape h = {};
  SB_CHECK_CUDA(cudaMemcpyAsync(&h, shape, sizeof(h), cudaMemcpyDeviceToHost, st));
  SB_CHECK_CUDA(cudaStreamSynchronize(st));
  scratch_free(shape, st);
  if (h.status) {
    set_error("sb_spts_analyze: a level dependency wait timed out");
    return SB_ETIMEOUT;
  }
  p->solvable = h.lower_bad ? 0 : 1;
  p->nlevels = N ? h.top + 1 : 0;
  const int L = p->nlevels;
  // level_ptr = exclusive scan of the per-level counts
  SB_CHECK_CUDA(cudaMemsetAsync(p->level_ptr, 0, sizeof(int) * ((size_t)L + 1), st));
  level_hist<<<grid1(N), kT, 0, st>>>(p->level, N, p->level_ptr);
  SB_CHECK_LAUNCH("level_hist");
  if ((r = prim::exclusive_scan(p->level_ptr, p->level_ptr, L + 1, st))) return r;
  // stable counting sort of rows by level; scratch: sort buffers, then the
  // window layout's counts
  const int gmax = N / win::kGroup + L + 1;  // no more groups than this
  prim::RadixBuffers rb;
  void* mem = nullptr;
  const size_t kb = align256(sizeof(unsigned long long) * N), vb = align256(sizeof(unsigned) * N);
  const size_t gb = align256(sizeof(int) * ((size_t)gmax + 1));
  const size_t lb = align256(sizeof(int) * ((size_t)L + 1));
  if ((r = scratch_alloc(&mem, 2 * kb + 2 * vb + lb + 2 * gb + 256, st))) return r;
  char* q = (char*)mem;
  rb.k[0] = (unsigned long long*)q;
  rb.k[1] = (unsigned long long*)(q + kb);
  rb.v[0] = (unsigned*)(q + 2 * kb);
  rb.v[1] = (unsigned*)(q + 2 * kb + vb);
  q += 2 * kb + 2 * vb;
  int* gstart = (int*)q;               // [L + 1] groups of the levels before
  int* glen = (int*)(q + lb);          // [gmax + 1] longest row of a group
  int* gbase = (int*)(q + lb + gb);    // [gmax + 1] first entry of a group
  win::Info* info = (win::Info*)(q + lb + 2 * gb);
  // where the window layout goes: the records in the memory of rcol and rval,
  // the group descriptors behind level_ptr's L + 1 entries if they fit there,
  // else at the end of rcol and rval
  long long cap = -1;  // 16-byte units for the records
  {
    const size_t area = align256(sizeof(int) * (size_t)nnz) + align256(sizeof(T) * (size_t)nnz);
    const size_t lp = align256(sizeof(int) * ((size_t)L + 1));
    const size_t slack = align256(sizeof(int) * ((size_t)N + 2)) - lp;
    const size_t gbytes = align256(sizeof(int4) * (size_t)gmax);
    size_t room = area;
    p->records = (char*)p->rcol;
    if (gbytes <= slack) {
      p->groups = (int4*)((char*)p->level_ptr + lp);
    } else if (gbytes < area) {
      room -= gbytes;
      p->groups = (int4*)(p->records + room);
    }
    if (p->groups) cap = std::min<long long>((long long)(room / 16), INT_MAX / 2);
  }
  int4* groups = cap >= 0 ? p->groups : nullptr;
  cudaError_t e = cudaMemsetAsync(gstart, 0, lb + 2 * gb + 256, st);
  if (e != cudaSuccess) r = cuda_status(e, "sb_spts_analyze");
  if (!r) {
    win::window_reach<<<grid1((long long)N + 1), kT, 0, st>>>(p->row_ptr, p->col, p->level,
                                                              p->level_ptr, N, L, gstart, info);
    e = cudaGetLastError();
    if (e != cudaSuccess) r = cuda_status(e, "window_reach");
    if (!r) r = prim::exclusive_scan(gstart, gstart, L + 1, st);
  }
  if (!r) {
    level_keys<<<grid1(N), kT, 0, st>>>(p->level, N, rb.k[0], rb.v[0]);
    e = cudaGetLastError();
    if (e != cudaSuccess) r = cuda_status(e, "level_keys");
  }
  const int ranges[2] = {0, prim::bits_for(L - 1)};
  int which = 0;
  if (!r) r = prim::radix_sort_ranges(rb, N, ranges, 1, &which, st);
  if (!r) {
    perm_order<<<grid1(N), kT, 0, st>>>(rb.v[which], N, p->perm, p->order);
    e = cudaGetLastError();
    if (e != cudaSuccess) r = cuda_status(e, "perm_order");
  }
  if (!r) {
    // row lengths in level order, scanned into rrow
    int* lens = (int*)rb.k[0];
    win::window_lengths<<<grid1((long long)N + 1), kT, 0, st>>>(p->row_ptr, p->perm, p->level, p->level_ptr,
                                                 gstart, N, lens, groups, glen);
    e = cudaGetLastError();
    if (e != cudaSuccess) r = cuda_status(e, "window_lengths");
    if (!r) r = prim::exclusive_scan(lens, p->rrow, (long long)N + 1, st);
    if (!r && groups) {
      win::window_sizes<<<grid1(gmax + 1), kT, 0, st>>>(groups, glen, gmax, gstart + L,
                                                        sizeof(T), gbase, info);
      e = cudaGetLastError();
      if (e != cudaSuccess) r = cuda_status(e, "window_sizes");
      if (!r) r = prim::exclusive_scan(gbase, gbase, gmax + 1, st);
      if (!r) {
        win::window_fill<T><<<grid1(N), kT, 0, st>>>(
            p->row_ptr, p->col, (const T*)p->val, p->perm, p->order, p->level, p->level_ptr, gstart,
            glen, gbase, N, L, cap, h.lower_bad == 0, info, groups, p->records);
        e = cudaGetLastError();
        if (e != cudaSuccess) r = cuda_status(e, "window_fill");
      }
    }
    if (!r) {
      reorder_rows<T><<<grid1(N), kT, 0, st>>>(p->row_ptr, p->col, (const T*)p->val, p->perm,
                                                p->order, p->rrow, N, info, p->rcol, (T*)p->rval);
      e = cudaGetLastError();
      if (e != cudaSuccess) r = cuda_status(e, "reorder_rows");
    }
  }
  if (!r) {
    e = cudaEventRecord(p->ev[1], st);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(&p->window, info, sizeof(win::Info), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e == cudaSuccess) e = cudaEventElapsedTime(&p->analysis_ms, p->ev[0], p->ev[1]);
    if (e != cudaSuccess) r = cuda_status(e, "sb_spts_analyze");
  }
  scratch_free(mem, st);
  return r;
}

template <typename T>
static win::View<T> window_view(const sb_spts_plan* p, T* yw) {
  return {p->groups,         p->records,     yw, p->window.ngroups, p->window.window,
          p->window.kmax, p->window.widest};
}

template <typename T, typename A, int KU>
static int launch_window(const sb_spts_plan* p, T* yw, int* status, cudaStream_t st) {
  auto k = win::window_solve<T, A, KU>;
  SB_CHECK_CUDA(cudaFuncSetAttribute((const void*)k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     win::kSmem));
  k<<<1, 32 * win::Warps<T, KU>::n, win::smem_bytes(p->window.window, sizeof(T)), st>>>(
      window_view(p, yw), status);
  SB_CHECK_LAUNCH("window_solve");
  return SB_OK;
}

// b into level order, the solve on one block, y back into natural order.
template <typename T, typename A>
static int solve_window(const sb_spts_plan* p, const T* b, T* y, int* status, cudaStream_t st) {
  const int N = p->N;
  T* yw = (T*)p->ywork;
  win::gather_by_perm<T><<<grid1(N), kT, 0, st>>>(b, p->perm, N, yw);
  SB_CHECK_LAUNCH("gather_by_perm");
  const int u = win::unroll_of(p->window.kmax);
  const int r = u == 4   ? launch_window<T, A, 4>(p, yw, status, st)
                : u == 8 ? launch_window<T, A, 8>(p, yw, status, st)
                         : launch_window<T, A, 16>(p, yw, status, st);
  if (r) return r;
  win::scatter_by_perm<T><<<grid1(N), kT, 0, st>>>(yw, p->perm, N, y);
  SB_CHECK_LAUNCH("scatter_by_perm");
  return SB_OK;
}

template <typename T, typename A>
static int solve_impl(const sb_spts_plan* p, int algo, const T* b, T* y, long long limit,
                      cudaStream_t st) {
  const int N = p->N;
  int* status = device_status_word();
  if (!status) {
    set_error("sb_spts_solve: device status word unavailable");
    return SB_ENOMEM;
  }
  if (algo != SB_SPTS_SYNCFREE && p->window.use)
    return solve_window<T, A>(p, b, y, status, st);
  T* yw = (T*)p->ywork;
  if (algo != SB_SPTS_SYNCFREE && p->nlevels <= kFewLevels) {
    for (int l = 0; l < p->nlevels; ++l) {
      spts_level_rows<T, A><<<grid1(p->window.rows), kT, 0, st>>>(
          p->rrow, p->rcol, (const T*)p->rval, p->level_ptr, l, p->perm, b, yw, y);
      SB_CHECK_LAUNCH("spts_level_rows");
    }
    return SB_OK;
  }
  if (algo == SB_SPTS_LEVEL && p->window.rows <= kLevelBlock) {
    // the two-round prefetch except for FP32 sums, where the one-round form
    // measured faster (1M-row random factor, 3470 levels: 6.54 against 7.27
    // ms; FP64 10.2 -> 9.40 ms with two rounds)
    constexpr bool two = !(sizeof(T) == 4 && sizeof(A) == 4);
    spts_level_block<T, A, two><<<1, kLevelBlock, 0, st>>>(
        p->rrow, p->rcol, (const T*)p->rval, p->level_ptr, p->nlevels, p->perm, b, yw, y);
    SB_CHECK_LAUNCH("spts_level_block");
    return SB_OK;
  }
  // pending values, and the ticket behind them, in one call
  SB_CHECK_CUDA(cudaMemsetAsync(yw, 0xff, (size_t)((char*)(p->ticket + 1) - (char*)yw), st));
  if (algo == SB_SPTS_SYNCFREE) {
    auto k = spts_syncfree_plan_rows<T, A>;
    k<<<polling_grid((const void*)k, algo, N, p->nlevels), kT, 0, st>>>(
        p->row_ptr, p->col, (const T*)p->val, N, b, yw, y, p->ticket, limit, status);
    SB_CHECK_LAUNCH("spts_syncfree_plan_rows");
  } else {
    auto k = spts_hybrid_rows<T, A>;
    k<<<polling_grid((const void*)k, algo, N, p->nlevels), kT, 0, st>>>(
        p->rrow, p->rcol, (const T*)p->rval, N, p->perm, b, yw, y, p->ticket, limit, status);
    SB_CHECK_LAUNCH("spts_hybrid_rows");
  }
  return SB_OK;
}

// ------------------------------------------------------------ no-allocation variant
// Scratch of sb_spts_syncfree_csr_noalloc: one ready flag per row for up to
// kNoAllocMaxRows rows, then the row ticket and the status word on their own
// 128-byte lines.  It is a file-scope device array, so every GPU that loads
// this library holds these 16 MiB until the process exits, and every call
// shares them.
constexpr int kNoAllocMaxRows = 1 << 22;  // 4,194,304 rows
constexpr int kNoAllocTail = 64;          // ticket at +0, status at +32 (words)
static __device__ __align__(256) unsigned g_noalloc_scratch[kNoAllocMaxRows + kNoAllocTail];

// Device address of g_noalloc_scratch for the current device, looked up once
// per device (with that device current) and cached.  The host-side symbol is
// only a stand-in and must never be handed to a kernel.
static unsigned* noalloc_scratch(int* status) {
  static std::mutex mu;
  static unsigned* addr[64] = {nullptr};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= 64) {
    *status = cuda_status(e == cudaSuccess ? cudaErrorInvalidDevice : e, "cudaGetDevice");
    return nullptr;
  }
  std::lock_guard<std::mutex> lk(mu);
  if (!addr[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) {
      *status = cuda_status(e, "cudaGetSymbolAddress(g_noalloc_scratch)");
      return nullptr;
    }
    addr[dev] = (unsigned*)p;
  }
  return addr[dev];
}

}  // namespace sb

using namespace sb;

// A batch's solves run in two branches of one graph, after one copy of the
// descriptors and counters: the plans with a window layout, each on one block,
// and the others with ready flags over the whole GPU.  A branch without solves
// is disabled for the run.
struct sb_spts_batch {
  int dtype = 0;
  int policy = 0;
  int capacity = 0;
  int device = 0;
  char* h = nullptr;             // pinned staging of everything below...
  char* d = nullptr;             // ...and its device copy
  size_t bytes = 0;
  // offsets into them
  size_t items = 0, sched = 0, order = 0, seg = 0, tickets = 0, work = 0;  // ready flags
  size_t views = 0, moves = 0, count = 0;                                  // windows
  int persistent = 0;            // capped grid: blocks per SM (0 = one warp per slot)
  cudaGraph_t graph_def = nullptr;
  cudaGraphExec_t graph = nullptr;
  cudaGraphNode_t reset_node = nullptr, solve_node = nullptr;
  cudaGraphNode_t gather_node = nullptr, window_node = nullptr, scatter_node = nullptr;
  cudaKernelNodeParams solve_params = {}, gather_params = {}, window_params = {},
                       scatter_params = {};
  bool flags_on = true, windows_on = true;  // the branches as the graph has them
  // kernel arguments (device addresses)
  void *a_items = nullptr, *a_sched = nullptr, *a_order = nullptr, *a_seg = nullptr,
       *a_tickets = nullptr, *a_work = nullptr, *a_views = nullptr, *a_moves = nullptr,
       *a_count = nullptr;
  void* reset_args[2] = {};
  void* solve_args[9] = {};
  void* move_args[2] = {};
  void* window_args[3] = {};
  long long limit = 0;
  int* status = nullptr;
  cudaEvent_t done = nullptr;
  bool pending = false;
  int full_per_sm = 1;     // resident blocks per SM of the solve kernel without a cap
  int smem_per_sm = 0;     // shared memory of an SM, bytes
  int smem_reserved = 0;   // shared memory the runtime reserves per block
  int smem_optin = 0;      // largest dynamic shared memory a block may request
};

static void spts_batch_release(sb_spts_batch* e) {
  if (e->graph) cudaGraphExecDestroy(e->graph);
  if (e->graph_def) cudaGraphDestroy(e->graph_def);
  if (e->done) cudaEventDestroy(e->done);
  if (e->h) cudaFreeHost(e->h);
  device_free(e->d);
  delete e;
}

template <typename T, typename A>
static const void* window_many(int u) {
  return u == 4   ? (const void*)win::window_solve_many<T, A, 4>
         : u == 8 ? (const void*)win::window_solve_many<T, A, 8>
                  : (const void*)win::window_solve_many<T, A, 16>;
}
static const void* window_kernel_for(int dtype, int policy, int u) {
  if (dtype == SB_F64) return window_many<double, double>(u);
  if (policy == SB_SPTS_ACC_F64) return window_many<float, double>(u);
  return window_many<float, float>(u);
}
static int window_threads(int dtype, int u) {
  return 32 * (u == 4   ? win::Warps<float, 4>::n
               : u == 8 ? (dtype == SB_F64 ? win::Warps<double, 8>::n : win::Warps<float, 8>::n)
                        : win::Warps<float, 16>::n);
}
static_assert(win::Warps<float, 4>::n == win::Warps<double, 4>::n &&
                  win::Warps<float, 16>::n == win::Warps<double, 16>::n,
              "window_threads takes these from the FP32 form");

static const void* spts_batch_kernel_for(int dtype, int policy) {
  if (dtype == SB_F64) return (const void*)spts_batch_kernel<double, double>;
  if (policy == SB_SPTS_ACC_F64) return (const void*)spts_batch_kernel<float, double>;
  return (const void*)spts_batch_kernel<float, float>;
}

// Descriptors and launch shapes of the items whose plans have a window layout
// (the longest solves first, so that the last blocks to finish are short);
// returns their number.
template <typename T>
static int stage_windows(sb_spts_batch* e, const sb_spts_batch_item* items, int n) {
  std::vector<std::pair<long long, int>> by_time;  // estimated ns, item
  int u = 4, window = 0;
  for (int i = 0; i < n; ++i) {
    const sb_spts_plan* p = items[i].plan;
    if (p->N == 0 || !p->window.use) continue;
    const int pu = win::unroll_of(p->window.kmax);
    u = std::max(u, pu);
    window = std::max(window, p->window.window);
    by_time.push_back({std::max(200LL * p->nlevels, (pu == 4 ? 26LL : pu == 8 ? 45 : 90) *
                                                        p->window.ngroups), i});
  }
  std::sort(by_time.rbegin(), by_time.rend());
  const int nw = (int)by_time.size();
  win::View<T>* views = (win::View<T>*)(e->h + e->views);
  win::Move<T>* moves = (win::Move<T>*)(e->h + e->moves);
  long long blocks = 0;
  for (int k = 0; k < nw; ++k) {
    const sb_spts_batch_item& it = items[by_time[k].second];
    T* yw = (T*)(it.work ? it.work : it.plan->ywork);
    views[k] = window_view<T>(it.plan, yw);
    moves[k] = {it.plan->perm, (const T*)it.b, yw, (T*)it.y, it.plan->N, (int)blocks};
    blocks += (it.plan->N + win::kMoveRows - 1) / win::kMoveRows;
  }
  *(int*)(e->h + e->count) = nw;
  e->gather_params.gridDim = e->scatter_params.gridDim =
      dim3((unsigned)std::max(1LL, blocks));
  e->window_params.func = const_cast<void*>(window_kernel_for(e->dtype, e->policy, u));
  e->window_params.blockDim = dim3(window_threads(e->dtype, u));
  e->window_params.gridDim = dim3(std::max(1, nw));
  long long smem = win::smem_bytes(window, sizeof(T));
  // a cap of k blocks per SM: more than 1/(k + 1) of its shared memory each
  if (e->persistent > 0)
    smem = std::max(smem, std::min<long long>(win::kSmem, e->smem_per_sm / (e->persistent + 1)));
  e->window_params.sharedMemBytes = (unsigned)smem;
  return nw;
}

// The same for the nf items that are solved with ready flags.
static int stage_flags(sb_spts_batch* e, const sb_spts_batch_item* items, int n, int nf) {
  SptsDesc* h_items = (SptsDesc*)(e->h + e->items);
  int* h_order = (int*)(e->h + e->order);
  long long* h_seg = (long long*)(e->h + e->seg);
  SptsSched* h_sched = (SptsSched*)(e->h + e->sched);
  std::vector<std::pair<int, int>> by_chunks;
  for (int i = 0; i < n; ++i) {
    const sb_spts_plan* p = items[i].plan;
    if (p->N > 0 && p->window.use) continue;
    const int k = (int)by_chunks.size();
    SptsDesc& d = h_items[k];
    d.rrow = p->rrow;
    d.rcol = p->rcol;
    d.rval = p->rval;
    d.perm = p->perm;
    d.yw = items[i].work ? items[i].work : p->ywork;
    d.b = items[i].b;
    d.y = items[i].y;
    d.N = p->N;
    d.pad = 0;
    by_chunks.push_back({(p->N + 31) / 32, k});
  }
  std::sort(by_chunks.begin(), by_chunks.end());
  long long warps = 0;
  int prev = 0;
  for (int k = 0; k < nf; ++k) {
    h_order[k] = by_chunks[k].second;
    h_seg[k] = warps;
    warps += (long long)(by_chunks[k].first - prev) * (nf - k);
    prev = by_chunks[k].first;
  }
  h_seg[nf] = warps;
  h_sched->M = nf;
  h_sched->warps = warps;
  const long long per_block = kTB / 32;
  long long blocks = std::max(1LL, (warps + per_block - 1) / per_block);
  if (e->persistent > 0)
    blocks = std::min(blocks, (long long)std::min(e->persistent, e->full_per_sm) * sm_count());
  SB_REQUIRE(blocks <= 0x7fffffffLL, "sb_spts_batch_run: batch too large");
  e->solve_params.gridDim = dim3((unsigned)blocks);
  // Resident blocks per SM: one per 8 systems, up to the occupancy limit.
  // Every resident warp that holds rows ahead of its system's frontier
  // polls, so a batch of few systems runs faster with few blocks per SM and
  // a batch of many with all of them (measured on B200 with FP32 factors: one
  // of 100k rows 0.95 -> 0.52 ms at one block per SM, 64 of them 0.83 ms at
  // full occupancy and 1.73 ms at one block per SM).  The cap is dynamic
  // shared memory that the solve does not use, rounded down to whole KiB, kept
  // only where the occupancy query confirms at least one block still fits.
  unsigned smem = 0;
  const int bps = std::min(e->full_per_sm, std::max(1, (nf + 7) / 8));
  if (e->persistent == 0 && bps < e->full_per_sm && e->smem_per_sm > 0) {
    long long want = (long long)e->smem_per_sm / bps - e->smem_reserved;
    want = std::min<long long>(want, e->smem_optin) / 1024 * 1024;
    int fit = 0;
    if (want > 0 && cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                        &fit, e->solve_params.func, kTB, (size_t)want) == cudaSuccess &&
        fit >= 1)
      smem = (unsigned)want;
  }
  e->solve_params.sharedMemBytes = smem;
  SB_CHECK_CUDA(cudaGraphExecKernelNodeSetParams(e->graph, e->solve_node, &e->solve_params));
  return SB_OK;
}

extern "C" {

int sb_spts_plan_growth(const sb_spts_plan* plan, double* growth, void* stream) {
  SB_TRACE("sb_spts_plan_growth");
  SB_REQUIRE(plan && growth, "sb_spts_plan_growth: null argument");
  *growth = 0.0;
  if (plan->N == 0) return SB_OK;
  cudaStream_t st = as_stream(stream);
  unsigned long long* d = nullptr;
  int r = scratch_alloc((void**)&d, sizeof(unsigned long long), st);
  if (r) return r;
  SB_CHECK_CUDA(cudaMemsetAsync(d, 0, sizeof(unsigned long long), st));
  const unsigned g = std::min<unsigned>(grid1(plan->N), (unsigned)sm_count() * 8);
  if (plan->dtype == SB_F64)
    growth_kernel<double><<<g, kT, 0, st>>>(plan->row_ptr, (const double*)plan->val, plan->N, d);
  else
    growth_kernel<float><<<g, kT, 0, st>>>(plan->row_ptr, (const float*)plan->val, plan->N, d);
  SB_CHECK_LAUNCH("growth_kernel");
  unsigned long long h = 0;
  SB_CHECK_CUDA(cudaMemcpyAsync(&h, d, sizeof(h), cudaMemcpyDeviceToHost, st));
  SB_CHECK_CUDA(cudaStreamSynchronize(st));
  scratch_free(d, st);
  double v;
  memcpy(&v, &h, sizeof(v));
  *growth = v;
  return SB_OK;
}

int sb_spts_batch_create(int dtype, int policy, int32_t capacity, sb_spts_batch** out) {
  SB_TRACE("sb_spts_batch_create");
  SB_REQUIRE(out, "sb_spts_batch_create: null output");
  *out = nullptr;
  SB_REQUIRE(dtype == SB_F32 || dtype == SB_F64, "sb_spts_batch_create: dtype must be F32 or F64");
  SB_REQUIRE(policy == SB_SPTS_ACC_NATIVE || policy == SB_SPTS_ACC_F64,
             "sb_spts_batch_create: bad accumulation policy");
  SB_REQUIRE(capacity > 0, "sb_spts_batch_create: capacity must be positive");
  int r = ensure_device();
  if (r) return r;
  int* status = device_status_word();
  if (!status) {
    set_error("sb_spts_batch_create: device status word unavailable");
    return SB_ENOMEM;
  }
  sb_spts_batch* e = new sb_spts_batch();
  e->dtype = dtype;
  e->policy = dtype == SB_F64 ? SB_SPTS_ACC_F64 : policy;
  e->capacity = capacity;
  cudaGetDevice(&e->device);
  cudaError_t ce = cudaSuccess;
#define SB_E(call)                    \
  if ((ce = (call)) != cudaSuccess) { \
    r = cuda_status(ce, #call);       \
    spts_batch_release(e);            \
    return r;                         \
  }
  // one block of memory for all descriptors and counters, copied per run
  const size_t cap = (size_t)capacity;
  const size_t vsize = dtype == SB_F64 ? sizeof(win::View<double>) : sizeof(win::View<float>);
  const size_t msize = dtype == SB_F64 ? sizeof(win::Move<double>) : sizeof(win::Move<float>);
  auto part = [&](size_t bytes) {
    const size_t at = e->bytes;
    e->bytes += (bytes + 15) / 16 * 16;
    return at;
  };
  e->items = part(sizeof(SptsDesc) * cap);
  e->sched = part(sizeof(SptsSched));
  e->order = part(sizeof(int) * cap);
  e->seg = part(sizeof(long long) * (cap + 1));
  e->tickets = part(sizeof(int) * cap);
  e->work = part(sizeof(unsigned long long));
  e->views = part(vsize * cap);
  e->moves = part(msize * cap);
  e->count = part(sizeof(int));
  SB_E(cudaMallocHost(&e->h, e->bytes));
  if ((r = device_alloc((void**)&e->d, e->bytes))) {
    spts_batch_release(e);
    return r;
  }
  SB_E(cudaEventCreateWithFlags(&e->done, cudaEventDisableTiming));
  memset(e->h, 0, e->bytes);
  e->limit = kDefaultSpin;
  e->status = status;
  e->a_items = e->d + e->items;
  e->a_sched = e->d + e->sched;
  e->a_order = e->d + e->order;
  e->a_seg = e->d + e->seg;
  e->a_tickets = e->d + e->tickets;
  e->a_work = e->d + e->work;
  e->a_views = e->d + e->views;
  e->a_moves = e->d + e->moves;
  e->a_count = e->d + e->count;
  const bool f64 = dtype == SB_F64;
  cudaGraphNode_t copy_node = nullptr;
  SB_E(cudaGraphCreate(&e->graph_def, 0));
  SB_E(cudaGraphAddMemcpyNode1D(&copy_node, e->graph_def, nullptr, 0, e->d, e->h, e->bytes,
                                cudaMemcpyHostToDevice));
  auto kernel_node = [&](cudaGraphNode_t* node, cudaKernelNodeParams& kp, cudaGraphNode_t after,
                         const void* func, int blocks, int threads, void** args) {
    kp.func = const_cast<void*>(func);
    kp.gridDim = dim3(blocks);
    kp.blockDim = dim3(threads);
    kp.sharedMemBytes = 0;
    kp.kernelParams = args;
    kp.extra = nullptr;
    return cudaGraphAddKernelNode(node, e->graph_def, &after, 1, &kp);
  };
  // ready flags: work vectors to pending, the solve (its grid is set per run)
  const void* kern = spts_batch_kernel_for(dtype, e->policy);
  e->reset_args[0] = &e->a_items;
  e->reset_args[1] = &e->a_sched;
  e->solve_args[0] = &e->a_items;
  e->solve_args[1] = &e->a_sched;
  e->solve_args[2] = &e->a_order;
  e->solve_args[3] = &e->a_seg;
  e->solve_args[4] = &e->a_tickets;
  e->solve_args[5] = &e->limit;
  e->solve_args[6] = &e->status;
  e->solve_args[7] = &e->a_work;
  e->solve_args[8] = &e->persistent;
  cudaKernelNodeParams reset_params = {};
  SB_E(kernel_node(&e->reset_node, reset_params, copy_node,
                   f64 ? (const void*)spts_batch_reset<double>
                       : (const void*)spts_batch_reset<float>,
                   sm_count() * 4, kT, e->reset_args));
  SB_E(kernel_node(&e->solve_node, e->solve_params, e->reset_node, kern, 1, kTB, e->solve_args));
  // windows: b into level order, the solves, y back into natural order
  e->move_args[0] = &e->a_moves;
  e->move_args[1] = &e->a_count;
  e->window_args[0] = &e->a_views;
  e->window_args[1] = &e->a_count;
  e->window_args[2] = &e->status;
  SB_E(kernel_node(&e->gather_node, e->gather_params, copy_node,
                   f64 ? (const void*)win::window_move<double, false>
                       : (const void*)win::window_move<float, false>,
                   1, 256, e->move_args));
  SB_E(kernel_node(&e->window_node, e->window_params, e->gather_node,
                   window_kernel_for(dtype, e->policy, 4), 1, window_threads(dtype, 4),
                   e->window_args));
  SB_E(kernel_node(&e->scatter_node, e->scatter_params, e->window_node,
                   f64 ? (const void*)win::window_move<double, true>
                       : (const void*)win::window_move<float, true>,
                   1, 256, e->move_args));
  {
    // the windows' few large blocks are placed before the other branch's many
    // small ones, which would keep them off the SMs until they are through
    int least = 0, greatest = 0;
    SB_E(cudaDeviceGetStreamPriorityRange(&least, &greatest));
    cudaKernelNodeAttrValue v = {};
    v.priority = std::max(greatest, least - 1);
    for (cudaGraphNode_t nd : {e->gather_node, e->window_node})
      SB_E(cudaGraphKernelNodeSetAttribute(nd, cudaKernelNodeAttributePriority, &v));
  }
  for (int u : {4, 8, 16})
    SB_E(cudaFuncSetAttribute(window_kernel_for(dtype, e->policy, u),
                              cudaFuncAttributeMaxDynamicSharedMemorySize, win::kSmem));
  SB_E(cudaGraphInstantiate(&e->graph, e->graph_def, 0));
  // residency cap of the solve (see sb_spts_batch_run): dynamic shared memory
  // that no solve uses, requested only to limit the blocks per SM
  SB_E(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&e->full_per_sm, kern, kTB, 0));
  e->full_per_sm = std::max(1, e->full_per_sm);
  SB_E(cudaDeviceGetAttribute(&e->smem_per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor,
                              e->device));
  SB_E(cudaDeviceGetAttribute(&e->smem_reserved, cudaDevAttrReservedSharedMemoryPerBlock,
                              e->device));
  SB_E(cudaDeviceGetAttribute(&e->smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin,
                              e->device));
  SB_E(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, e->smem_optin));
#undef SB_E
  *out = e;
  return SB_OK;
}

int sb_spts_batch_set_grid(sb_spts_batch* e, int32_t blocks_per_sm) {
  SB_TRACE("sb_spts_batch_set_grid");
  SB_REQUIRE(e, "sb_spts_batch_set_grid: null executor");
  SB_REQUIRE(blocks_per_sm >= 0, "sb_spts_batch_set_grid: negative block count");
  if (e->pending) SB_CHECK_CUDA(cudaEventSynchronize(e->done));
  e->persistent = blocks_per_sm;
  return SB_OK;
}

int sb_spts_batch_destroy(sb_spts_batch* e) {
  SB_TRACE("sb_spts_batch_destroy");
  if (!e) return SB_OK;
  if (e->pending) cudaEventSynchronize(e->done);
  spts_batch_release(e);
  return SB_OK;
}

int sb_spts_batch_run(sb_spts_batch* e, const sb_spts_batch_item* items, int32_t n,
                      void* stream) {
  SB_TRACE("sb_spts_batch_run");
  SB_REQUIRE(e, "sb_spts_batch_run: null executor");
  SB_REQUIRE(n >= 0 && n <= e->capacity, "sb_spts_batch_run: %d items exceed capacity %d", n,
             e->capacity);
  SB_REQUIRE(n == 0 || items, "sb_spts_batch_run: null items");
  for (int i = 0; i < n; ++i) {
    const sb_spts_plan* p = items[i].plan;
    SB_REQUIRE(p, "sb_spts_batch_run: item %d: null plan", i);
    SB_REQUIRE(p->dtype == e->dtype, "sb_spts_batch_run: item %d: plan dtype differs", i);
    SB_REQUIRE(p->device == e->device, "sb_spts_batch_run: item %d: plan on another device", i);
    SB_REQUIRE(p->N == 0 || (items[i].b && items[i].y), "sb_spts_batch_run: item %d: null vector",
               i);
    if (p->N > 0 && !p->solvable) {
      set_error("sb_spts_batch_run: item %d: matrix is not lower triangular with its diagonal "
                "stored last", i);
      return SB_EINVAL;
    }
    const size_t vs = p->dtype == SB_F64 ? 8 : 4;
    SB_REQUIRE(reinterpret_cast<uintptr_t>(items[i].work) % vs == 0,
               "sb_spts_batch_run: item %d: work vector not aligned to the value size", i);
  }
  {
    // a plan's own work vector serves one solve per run
    std::vector<const sb_spts_plan*> ps;
    for (int i = 0; i < n; ++i)
      if (!items[i].work) ps.push_back(items[i].plan);
    std::sort(ps.begin(), ps.end());
    for (size_t i = 1; i < ps.size(); ++i)
      SB_REQUIRE(ps[i] != ps[i - 1],
                 "sb_spts_batch_run: a plan appears twice in one batch with its own work vector");
  }
  // the pinned staging buffer is read by the previous run's first node
  if (e->pending) SB_CHECK_CUDA(cudaEventSynchronize(e->done));
  cudaStream_t st = as_stream(stream);
  const int nw = e->dtype == SB_F64 ? stage_windows<double>(e, items, n)
                                    : stage_windows<float>(e, items, n);
  const int nf = n - nw;
  if (nw > 0) {
    SB_CHECK_CUDA(cudaGraphExecKernelNodeSetParams(e->graph, e->gather_node, &e->gather_params));
    SB_CHECK_CUDA(cudaGraphExecKernelNodeSetParams(e->graph, e->window_node, &e->window_params));
    SB_CHECK_CUDA(cudaGraphExecKernelNodeSetParams(e->graph, e->scatter_node, &e->scatter_params));
  }
  if (nf > 0) {
    const int r = stage_flags(e, items, n, nf);
    if (r) return r;
  }
  if ((nw > 0) != e->windows_on) {
    for (cudaGraphNode_t nd : {e->gather_node, e->window_node, e->scatter_node})
      SB_CHECK_CUDA(cudaGraphNodeSetEnabled(e->graph, nd, nw > 0));
    e->windows_on = nw > 0;
  }
  if ((nf > 0) != e->flags_on) {
    for (cudaGraphNode_t nd : {e->reset_node, e->solve_node})
      SB_CHECK_CUDA(cudaGraphNodeSetEnabled(e->graph, nd, nf > 0));
    e->flags_on = nf > 0;
  }
  SB_CHECK_CUDA(cudaGraphLaunch(e->graph, st));
  SB_CHECK_CUDA(cudaEventRecord(e->done, st));
  e->pending = true;
  return SB_OK;
}

int sb_spts_syncfree_csr_noalloc(int dtype, const int32_t* row_ptr, const int32_t* col,
                                 const void* val, int32_t N, const void* b, void* y,
                                 int64_t spin_limit_cycles, void* stream) {
  SB_TRACE("sb_spts_syncfree_csr_noalloc");
  SB_REQUIRE(dtype == SB_F32 || dtype == SB_F64, "sb_spts_syncfree_csr_noalloc: bad dtype");
  SB_REQUIRE(N >= 0, "sb_spts_syncfree_csr_noalloc: negative size");
  if (N > kNoAllocMaxRows) {
    set_error("sb_spts_syncfree_csr_noalloc: N = %d exceeds the fixed scratch limit of %d rows "
              "(use sb_spts_syncfree_csr)", N, kNoAllocMaxRows);
    return SB_EINVAL;
  }
  if (N == 0) return SB_OK;
  SB_REQUIRE(row_ptr && col && val && b && y, "sb_spts_syncfree_csr_noalloc: null pointer");
  int r = ensure_device();
  if (r) return r;
  unsigned* scratch = noalloc_scratch(&r);
  if (!scratch) return r;
  cudaStream_t st = as_stream(stream);
  unsigned* flags = scratch;
  int* ticket = (int*)(scratch + kNoAllocMaxRows);
  int* status = (int*)(scratch + kNoAllocMaxRows + 32);
  // the array keeps the previous call's contents: clear what must start at 0
  SB_CHECK_CUDA(cudaMemsetAsync(flags, 0, sizeof(unsigned) * (size_t)N, st));
  SB_CHECK_CUDA(cudaMemsetAsync(ticket, 0, sizeof(unsigned) * kNoAllocTail, st));
  const long long limit = spin_limit_cycles > 0 ? spin_limit_cycles : kDefaultSpin;
  if (dtype == SB_F64) {
    auto k = spts_syncfree_rows<double, double>;
    k<<<natural_order_grid((const void*)k), kT, 0, st>>>(row_ptr, col, (const double*)val, N,
                                                          (const double*)b, (double*)y, flags,
                                                          ticket, limit, status);
  } else {
    auto k = spts_syncfree_rows<float, float>;
    k<<<natural_order_grid((const void*)k), kT, 0, st>>>(row_ptr, col, (const float*)val, N,
                                                          (const float*)b, (float*)y, flags,
                                                          ticket, limit, status);
  }
  SB_CHECK_LAUNCH("spts_syncfree_rows");
  int dstat = 0;
  SB_CHECK_CUDA(cudaMemcpyAsync(&dstat, status, sizeof(int), cudaMemcpyDeviceToHost, st));
  SB_CHECK_CUDA(cudaStreamSynchronize(st));
  if (dstat) {
    set_error("sb_spts_syncfree_csr_noalloc: a dependency wait ran out (row never became ready)");
    return SB_ETIMEOUT;
  }
  return SB_OK;
}

int sb_spts_analyze(int dtype, const int32_t* row_ptr, const int32_t* col, const void* val,
                    int32_t N, int64_t nnz, void* stream, sb_spts_plan** plan) {
  SB_TRACE("sb_spts_analyze");
  SB_REQUIRE(plan, "sb_spts_analyze: null plan output");
  *plan = nullptr;
  SB_REQUIRE(dtype == SB_F32 || dtype == SB_F64, "sb_spts_analyze: dtype must be F32 or F64");
  SB_REQUIRE(N >= 0 && nnz >= 0 && nnz <= 0x7fffffffLL, "sb_spts_analyze: bad size");
  SB_REQUIRE(row_ptr && (nnz == 0 || (col && val)), "sb_spts_analyze: null pointer");
  int r = ensure_device();
  if (r) return r;
  sb_spts_plan* p = new sb_spts_plan();
  p->dtype = dtype;
  p->N = N;
  p->nnz = nnz;
  p->row_ptr = row_ptr;
  p->col = col;
  p->val = val;
  cudaGetDevice(&p->device);
  cudaStream_t st = as_stream(stream);
  if (N == 0) {
    *plan = p;
    return SB_OK;
  }
  r = dtype == SB_F32 ? analyze_impl<float>(p, st) : analyze_impl<double>(p, st);
  if (r) {
    cudaStreamSynchronize(st);
    plan_release(p);
    delete p;
    return r;
  }
  *plan = p;
  return SB_OK;
}

int sb_spts_plan_destroy(sb_spts_plan* plan) {
  SB_TRACE("sb_spts_plan_destroy");
  if (!plan) return SB_OK;
  cudaDeviceSynchronize();
  plan_release(plan);
  delete plan;
  return SB_OK;
}

int sb_spts_plan_info(const sb_spts_plan* plan, int32_t* nlevels, int32_t* solvable) {
  SB_TRACE("sb_spts_plan_info");
  SB_REQUIRE(plan && nlevels && solvable, "sb_spts_plan_info: null argument");
  *nlevels = plan->nlevels;
  *solvable = plan->solvable;
  return SB_OK;
}

int sb_spts_plan_analysis_ms(const sb_spts_plan* plan, float* ms) {
  SB_TRACE("sb_spts_plan_analysis_ms");
  SB_REQUIRE(plan && ms, "sb_spts_plan_analysis_ms: null argument");
  *ms = plan->analysis_ms;
  return SB_OK;
}

int sb_spts_plan_levels(const sb_spts_plan* plan, int32_t* level, int32_t* level_ptr,
                        int32_t* permutation, int32_t* order, void* stream) {
  SB_TRACE("sb_spts_plan_levels");
  SB_REQUIRE(plan, "sb_spts_plan_levels: null plan");
  const size_t n = sizeof(int) * (size_t)plan->N;
  cudaStream_t st = as_stream(stream);
  if (plan->N == 0) return SB_OK;
  if (level) SB_CHECK_CUDA(cudaMemcpyAsync(level, plan->level, n, cudaMemcpyDeviceToDevice, st));
  if (level_ptr)
    SB_CHECK_CUDA(cudaMemcpyAsync(level_ptr, plan->level_ptr,
                                  sizeof(int) * ((size_t)plan->nlevels + 1),
                                  cudaMemcpyDeviceToDevice, st));
  if (permutation)
    SB_CHECK_CUDA(cudaMemcpyAsync(permutation, plan->perm, n, cudaMemcpyDeviceToDevice, st));
  if (order) SB_CHECK_CUDA(cudaMemcpyAsync(order, plan->order, n, cudaMemcpyDeviceToDevice, st));
  return SB_OK;
}

int sb_spts_plan_reordered(const sb_spts_plan* plan, int32_t* row_ptr, int32_t* col, void* val,
                           void* stream) {
  SB_TRACE("sb_spts_plan_reordered");
  SB_REQUIRE(plan, "sb_spts_plan_reordered: null plan");
  cudaStream_t st = as_stream(stream);
  if (plan->N == 0) return SB_OK;
  if (row_ptr)
    SB_CHECK_CUDA(cudaMemcpyAsync(row_ptr, plan->rrow, sizeof(int) * ((size_t)plan->N + 1),
                                  cudaMemcpyDeviceToDevice, st));
  if (plan->window.use && (col || val)) {
    const unsigned g = grid1(32LL * plan->window.ngroups);
    if (plan->dtype == SB_F64)
      win::window_to_csr<double><<<g, kT, 0, st>>>(plan->rrow, plan->level_ptr, plan->groups,
                                                   plan->window.ngroups, plan->window.window,
                                                   plan->records, col, (double*)val);
    else
      win::window_to_csr<float><<<g, kT, 0, st>>>(plan->rrow, plan->level_ptr, plan->groups,
                                                  plan->window.ngroups, plan->window.window,
                                                  plan->records, col, (float*)val);
    SB_CHECK_LAUNCH("window_to_csr");
    return SB_OK;
  }
  if (col)
    SB_CHECK_CUDA(cudaMemcpyAsync(col, plan->rcol, sizeof(int) * (size_t)plan->nnz,
                                  cudaMemcpyDeviceToDevice, st));
  if (val)
    SB_CHECK_CUDA(cudaMemcpyAsync(val, plan->rval, dtype_size(plan->dtype) * (size_t)plan->nnz,
                                  cudaMemcpyDeviceToDevice, st));
  return SB_OK;
}

int sb_spts_solve(const sb_spts_plan* plan, int algo, int policy, const void* b, void* y,
                  void* stream) {
  SB_TRACE("sb_spts_solve");
  SB_REQUIRE(plan, "sb_spts_solve: null plan");
  SB_REQUIRE(algo == SB_SPTS_LEVEL || algo == SB_SPTS_SYNCFREE || algo == SB_SPTS_HYBRID,
             "sb_spts_solve: unknown algorithm %d", algo);
  if (plan->N == 0) return SB_OK;
  SB_REQUIRE(b && y, "sb_spts_solve: null vector");
  if (!plan->solvable) {
    set_error("sb_spts_solve: matrix is not lower triangular with its diagonal stored last");
    return SB_EINVAL;
  }
  cudaStream_t st = as_stream(stream);
  if (plan->dtype == SB_F64)
    return solve_impl<double, double>(plan, algo, (const double*)b, (double*)y, kDefaultSpin, st);
  if (policy == SB_SPTS_ACC_F64)
    return solve_impl<float, double>(plan, algo, (const float*)b, (float*)y, kDefaultSpin, st);
  return solve_impl<float, float>(plan, algo, (const float*)b, (float*)y, kDefaultSpin, st);
}

int sb_spts_syncfree_csr(int dtype, const int32_t* row_ptr, const int32_t* col, const void* val,
                         int32_t N, const void* b, void* y, int64_t spin_limit_cycles,
                         void* stream) {
  SB_TRACE("sb_spts_syncfree_csr");
  SB_REQUIRE(dtype == SB_F32 || dtype == SB_F64, "sb_spts_syncfree_csr: bad dtype");
  SB_REQUIRE(N >= 0, "sb_spts_syncfree_csr: negative size");
  if (N == 0) return SB_OK;
  SB_REQUIRE(row_ptr && col && val && b && y, "sb_spts_syncfree_csr: null pointer");
  int r = ensure_device();
  if (r) return r;
  cudaStream_t st = as_stream(stream);
  int* status = device_status_word();
  if (!status) return SB_ENOMEM;
  unsigned* flags = nullptr;
  if ((r = scratch_alloc((void**)&flags, sizeof(unsigned) * ((size_t)N + 8), st))) return r;
  int* ticket = (int*)(flags + N);
  SB_CHECK_CUDA(cudaMemsetAsync(flags, 0, sizeof(unsigned) * ((size_t)N + 8), st));
  const long long limit = spin_limit_cycles > 0 ? spin_limit_cycles : kDefaultSpin;
  if (dtype == SB_F64) {
    auto k = spts_syncfree_rows<double, double>;
    k<<<natural_order_grid((const void*)k), kT, 0, st>>>(row_ptr, col, (const double*)val, N,
                                                     (const double*)b, (double*)y, flags, ticket,
                                                     limit, status);
  } else {
    auto k = spts_syncfree_rows<float, float>;
    k<<<natural_order_grid((const void*)k), kT, 0, st>>>(row_ptr, col, (const float*)val, N,
                                                     (const float*)b, (float*)y, flags, ticket,
                                                     limit, status);
  }
  SB_CHECK_LAUNCH("spts_syncfree_rows");
  int dstat = 0;
  SB_CHECK_CUDA(cudaMemcpyAsync(&dstat, status, sizeof(int), cudaMemcpyDeviceToHost, st));
  SB_CHECK_CUDA(cudaStreamSynchronize(st));
  scratch_free(flags, st);
  if (dstat) {
    SB_CHECK_CUDA(cudaMemset(status, 0, sizeof(int)));
    set_error("sb_spts_syncfree_csr: a dependency wait ran out (row never became ready)");
    return SB_ETIMEOUT;
  }
  return SB_OK;
}

int sb_spts_csc(int dtype, const int32_t* col_ptr, const int32_t* row, const void* val,
                int32_t N, int64_t nnz, const void* x, void* y, void* stream) {
  SB_TRACE("sb_spts_csc");
  SB_REQUIRE(dtype == SB_F32 || dtype == SB_F64, "sb_spts_csc: dtype must be F32 or F64");
  SB_REQUIRE(N >= 0 && nnz >= 0 && nnz <= 0x7fffffffLL, "sb_spts_csc: bad size");
  if (N == 0) return SB_OK;
  SB_REQUIRE(col_ptr && row && val && x && y, "sb_spts_csc: null pointer");
  int r = ensure_device();
  if (r) return r;
  cudaStream_t st = as_stream(stream);
  const size_t vb = dtype_size(dtype);
  void* mem = nullptr;
  // [flag] [CSR row_ptr N+1] [CSR col nnz] [CSR val nnz]
  const size_t off_rp = 16, off_col = off_rp + sizeof(int) * ((size_t)N + 1);
  const size_t off_val = (off_col + sizeof(int) * (size_t)nnz + 15) / 16 * 16;
  if ((r = scratch_alloc(&mem, off_val + vb * (size_t)nnz, st))) return r;
  char* p = (char*)mem;
  int* flag = (int*)p;
  int* rp = (int*)(p + off_rp);
  int* col = (int*)(p + off_col);
  void* cval = p + off_val;
  SB_CHECK_CUDA(cudaMemsetAsync(flag, 0, sizeof(int), st));
  csc_lower_check<<<grid1(N), kT, 0, st>>>(col_ptr, row, N, flag);
  SB_CHECK_LAUNCH("csc_lower_check");
  int h = 0;
  SB_CHECK_CUDA(cudaMemcpyAsync(&h, flag, sizeof(int), cudaMemcpyDeviceToHost, st));
  SB_CHECK_CUDA(cudaStreamSynchronize(st));
  if (h) {
    scratch_free(mem, st);
    set_error("sb_spts_csc: every column must start with its diagonal, the other rows below it");
    return SB_EINVAL;
  }
  // the CSC arrays are the CSR of L^T; its transpose is L in CSR with each
  // row's entries in increasing column order (diagonal last)
  r = sb_transpose_csr(dtype, col_ptr, row, val, N, nnz, rp, col, cval, stream);
  if (!r) r = sb_spts_syncfree_csr(dtype, rp, col, cval, N, x, y, 0, stream);
  scratch_free(mem, st);
  return r;
}

}  // extern "C"
