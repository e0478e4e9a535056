// sb_spts_window.cuh -- triangular solves whose dependencies all lie in a
// window of recently solved rows held in shared memory.
//
// The solves are bound by the chain of levels.  With ready flags a row's value
// goes from SM to SM through L2 (a store, the poll that sees it, the gather:
// 1.26 us per level on B200 whatever the level's width), and a barrier per
// level with the values in L2 costs more.  Here one block solves the whole
// factor with the values of the last W rows in a shared-memory ring: a
// dependency is a shared-memory read, and an mbarrier closes a level (0.16 us
// per level FP32, 0.20 FP64 on narrow levels).  Measured (solve with its two
// passes for b and y; level / hybrid before -> now): 1M-row random factor of
// 3481 levels FP64 9.26 / 4.71 -> 1.70 ms, FP32 6.53 / 3.97 -> 1.21; 100k rows
// in 3044 levels FP64 3.07 / 3.97 -> 0.61; 3-D Laplacian 24^3 FP32 0.074 /
// 0.076 -> 0.030; 24 factors of up to 1M rows in one batch 5.24 -> 1.59.  Wide
// levels stay with the ready flags (window_decide).
//
// With several groups per level the block is bound by its own instructions
// (a warp takes about 1500 cycles for a group of 32 rows), so the layout is
// made for few of them: rows in level order are cut into groups of up to 32
// rows of one level; a group's record holds its rows' values in pairs and the
// columns as the 16-bit ring slots of the rows they name, in quads, lane by
// lane, so that a row of 7 entries takes six wide loads and no address
// arithmetic (thread-per-row loads of CSR rows: one line per lane and load;
// one value per load: 2.66 ms for the FP64 factor above).  Bulk copies into
// shared memory ahead of the registers (2.71 ms), a shared-memory counter with
// fences instead of the mbarriers (3.0 ms), a block barrier per level (4.2 ms),
// clusters of 2 to 8 blocks with the values stored to every block's ring
// (4.1 ms; 64^3 Laplacian 0.29 ms against 0.25) and a division prepared by the
// reciprocal (no gain) were measured and left out.
//
// Arithmetic is the row kernel's (t = 0; t += L_ij * y_j in storage order,
// separately rounded; y_i = (b_i - t) / L_ii), so the bits are those of the
// level-set and hybrid solves.
#pragma once

#include <climits>

#include "sb_common.cuh"

namespace sb {

template <typename T> __device__ __forceinline__ T mul_rn(T a, T b);
template <> __device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
template <> __device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
template <typename T> __device__ __forceinline__ T add_rn(T a, T b);
template <> __device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
template <> __device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
template <typename T> __device__ __forceinline__ T sub_rn(T a, T b);
template <> __device__ __forceinline__ float sub_rn(float a, float b) { return __fsub_rn(a, b); }
template <> __device__ __forceinline__ double sub_rn(double a, double b) { return __dsub_rn(a, b); }
template <typename T> __device__ __forceinline__ T div_rn(T a, T b);
template <> __device__ __forceinline__ float div_rn(float a, float b) { return __fdiv_rn(a, b); }
template <> __device__ __forceinline__ double div_rn(double a, double b) { return __ddiv_rn(a, b); }

namespace win {
namespace {

constexpr int kGroup = 32;                 // rows of a group at most: one warp
constexpr int kMaxK = 15;                  // off-diagonal entries of a row at most
constexpr int kMaxWarps = 32;              // warps of a solving block
constexpr int kLevelBars = 2 * kMaxWarps;
constexpr int kMaxArrivals = (1 << 20) - 1;  // of a barrier's phase
constexpr int kSmem = 225 * 1024;  // ring and stages, of the 227 KB a block may have

// Decision and sizes of a plan's window layout, on the device and then in the
// plan: use = 1 when the layout was built.
struct Info {
  int reach;   // rows from a dependency to the end of the level that reads it, at most
  int kmax;    // longest row, off-diagonal entries
  int use;
  int window;  // ring slots
  int widest;  // groups of a level at most
  int rows;    // rows of a level at most
  int ngroups;
  unsigned long long size16;  // 16-byte units of all group records, also where they
                              // are too many for the layout's 32-bit offsets
};

// A group: {first row, record offset in 16-byte units, level,
// rows | entries per row << 6 | arrivals on its level's barrier << 11}.
// Its record, for n rows of at most k off-diagonal entries: the diagonal and
// the entries' values, padded to an even number, as pairs (pair p of all rows
// before pair p + 1), then the entries' ring slots, padded to a multiple of
// four, as quads in the same manner: a lane reads its row with few wide loads.
__device__ __forceinline__ int group_rows(int4 g) { return g.w & 63; }
__device__ __forceinline__ int group_len(int4 g) { return (g.w >> 6) & 31; }
__device__ __forceinline__ uint32_t group_arrivals(int4 g) { return (unsigned)g.w >> 11; }
__host__ __device__ __forceinline__ int record_pairs(int k) { return (k + 2) / 2; }
__host__ __device__ __forceinline__ int record_quads(int k) { return (k + 3) / 4; }
// Bytes of the values, a multiple of 16; of the whole record in 16-byte units.
__host__ __device__ __forceinline__ int record_values(int n, int k, int tsize) {
  return (n * record_pairs(k) * 2 * tsize + 15) / 16 * 16;
}
__host__ __device__ __forceinline__ int record16(int n, int k, int tsize) {
  return (record_values(n, k, tsize) + n * record_quads(k) * 8 + 15) / 16;
}
__host__ __device__ __forceinline__ long long smem_bytes(int window, int tsize) {
  return (long long)(window + 1) * tsize;  // one slot more for absent entries
}

// ------------------------------------------------------------ building

// reach over all rows (natural order): from the first row of the lowest level
// a row reads to the end of its own level; and the groups of every level
// (cnt[nlevels + 1], to be scanned).  One thread per row, and one more.
__global__ void window_reach(const int* __restrict__ row_ptr, const int* __restrict__ col,
                             const int* __restrict__ level, const int* __restrict__ level_ptr,
                             int N, int nlevels, int* __restrict__ cnt, Info* __restrict__ info) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  int m = 0, rows = 0;
  if (i < N) {
    const int s = row_ptr[i], e = row_ptr[i + 1] - 1;
    int lo = INT_MAX;
    for (int j = s; j < e; ++j) {
      const int c = col[j];
      if (c >= 0 && c < i) lo = min(lo, __ldg(level + c));
    }
    if (lo != INT_MAX) m = level_ptr[level[i] + 1] - level_ptr[lo];
  }
  if (i < nlevels) rows = level_ptr[i + 1] - level_ptr[i];
  if (i <= nlevels) cnt[i] = (rows + kGroup - 1) / kGroup;
  m = __reduce_max_sync(0xffffffffu, m);
  rows = __reduce_max_sync(0xffffffffu, rows);
  if ((threadIdx.x & 31) == 0) {
    if (m > 0) atomicMax(&info->reach, m);
    if (rows > 0) {
      atomicMax(&info->rows, rows);
      atomicMax(&info->widest, (rows + kGroup - 1) / kGroup);
    }
  }
}

// Row lengths in level order (N + 1, to be scanned), and each group's longest
// row (off-diagonal).
__global__ void window_lengths(const int* __restrict__ row_ptr, const int* __restrict__ perm,
                               const int* __restrict__ level, const int* __restrict__ level_ptr,
                               const int* __restrict__ gstart, int N, int* __restrict__ lens,
                               int4* __restrict__ groups, int* __restrict__ glen) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p == N) lens[N] = 0;
  if (p >= N) return;
  const int src = perm[p];
  const int len = row_ptr[src + 1] - row_ptr[src];
  lens[p] = len;
  if (!groups) return;
  const int l = level[src], lp = level_ptr[l], i = p - lp;
  const int g = gstart[l] + i / kGroup;
  const unsigned m = __match_any_sync(__activemask(), g);
  const int k = __reduce_max_sync(m, len - 1);
  if ((int)(threadIdx.x & 31) == __ffs(m) - 1 && k > 0) atomicMax(glen + g, k);
  if (i % kGroup == 0)
    groups[g] = make_int4(p, 0, l, min(kGroup, level_ptr[l + 1] - p));
}

// Record sizes (n = the bound on the number of groups; those past the last
// have none), to be scanned; their total and the longest row into info.
__global__ void window_sizes(const int4* __restrict__ groups, const int* __restrict__ glen, int n,
                             const int* __restrict__ ngroups, int tsize, int* __restrict__ size,
                             Info* __restrict__ info) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  const bool in = g <= n && g < *ngroups;
  const int k = in ? glen[g] : 0;
  const int units = in ? record16(group_rows(groups[g]), min(k, kMaxK), tsize) : 0;
  if (g <= n) size[g] = units;
  const int sum = __reduce_add_sync(0xffffffffu, units), most = __reduce_max_sync(0xffffffffu, k);
  if ((threadIdx.x & 31) == 0) {
    if (sum) atomicAdd(&info->size16, (unsigned long long)sum);
    if (most > 0) atomicMax(&info->kmax, most);
  }
}

// Values of a row that the solve holds in registers (the diagonal and up to
// KU - 1 entries).
__host__ __device__ __forceinline__ int unroll_of(int kmax) {
  return kmax <= 3 ? 4 : kmax <= 7 ? 8 : 16;
}

// Whether to build the layout: it fits (cap: the record units there is room
// for, below 2^30, so that offsets into accepted ones fit in 32 bits, while the
// total can pass 2^31 from 215M FP64 rows on; lower: the structure the solves
// need), and one block with its window solves the factor faster than ready
// flags over the whole GPU.  A block takes a fixed time per group once a level
// has several, the ready flags a fixed time per level.  Measured on B200 (ns
// per group at KU 4 / 8 / 16: FP32 24 / 35 / 75, FP64 27 / 51 / 105; us per
// level of the ready flags: FP32 1.05-1.14, FP64 1.26-1.35), the two meet at
// about 40, 26 and 12 groups per level.
__host__ __device__ __forceinline__ int window_rows(int reach) {
  return reach > kGroup ? (reach + kGroup - 1) / kGroup * kGroup : kGroup;
}
__host__ __device__ __forceinline__ bool window_wins(const Info& f, int ngroups, int nlevels,
                                                     long long cap, int tsize, bool lower) {
  const int w = window_rows(f.reach), u = unroll_of(f.kmax);
  const int most = u == 4 ? 40 : u == 8 ? 26 : 12;
  return lower && f.reach < 0xffe0 && f.kmax <= kMaxK && (long long)f.size16 <= cap &&
         f.widest <= kMaxArrivals && smem_bytes(w, tsize) <= kSmem &&
         (long long)ngroups <= (long long)most * nlevels;
}

// Decides, completes the group descriptors and writes the records: one thread
// per row in level order.
template <typename T>
__global__ void window_fill(const int* __restrict__ row_ptr, const int* __restrict__ col,
                            const T* __restrict__ val, const int* __restrict__ perm,
                            const int* __restrict__ order, const int* __restrict__ level,
                            const int* __restrict__ level_ptr, const int* __restrict__ gstart,
                            const int* __restrict__ glen, const int* __restrict__ gbase, int N,
                            int nlevels, long long cap, bool lower, Info* info,
                            int4* __restrict__ groups, char* __restrict__ records) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= N) return;
  const bool use = window_wins(*info, gstart[nlevels], nlevels, cap, sizeof(T), lower);
  const int w = window_rows(info->reach);
  if (p == 0) {
    info->ngroups = gstart[nlevels];
    info->window = w;
    info->use = use;
  }
  if (!use) return;
  const int src = perm[p];
  const int l = level[src], i = p - level_ptr[l];
  const int g = gstart[l] + i / kGroup, lane = i % kGroup;
  const int n = min(kGroup, level_ptr[l + 1] - (p - lane));
  const int k = glen[g], base = gbase[g];
  if (lane == 0) {
    groups[g].y = base;
    const int missing = info->widest - (gstart[l + 1] - gstart[l]);
    groups[g].w = n | k << 6 | (int)((unsigned)(1 + (i == 0 ? missing : 0)) << 11);
  }
  char* rec = records + 16LL * base;
  T* v = reinterpret_cast<T*>(rec);
  unsigned short* sl = reinterpret_cast<unsigned short*>(rec + record_values(n, k, sizeof(T)));
  const int s = row_ptr[src], len = row_ptr[src + 1] - 1 - s;
  v[2 * lane] = val[s + len];
  for (int j = 0; j < 2 * record_pairs(k) - 1; ++j)
    v[((j + 1) / 2 * n + lane) * 2 + (j + 1) % 2] = j < len ? val[s + j] : T(0);
  for (int j = 0; j < 4 * record_quads(k); ++j)
    sl[(j / 4 * n + lane) * 4 + j % 4] = (unsigned short)(j < len ? order[col[s + j]] % w : w);
}

// The reordered CSR out of the window layout (rrow: its row pointers): a
// ring slot names the one row of the last `w` before the end of the reading
// row's level.
template <typename T>
__global__ void window_to_csr(const int* __restrict__ rrow, const int* __restrict__ level_ptr,
                              const int4* __restrict__ groups, int ngroups, int w,
                              const char* __restrict__ records, int* __restrict__ rcol,
                              T* __restrict__ rval) {
  const int lane = threadIdx.x & 31;
  const int g = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (g >= ngroups) return;
  const int4 d = groups[g];
  const int n = group_rows(d), k = group_len(d);
  if (lane >= n) return;
  const int p = d.x + lane;
  const int s = rrow[p], len = rrow[p + 1] - 1 - s;
  const int last = level_ptr[d.z + 1] - 1;  // the level's last row
  const char* rec = records + 16LL * d.y;
  const T* v = reinterpret_cast<const T*>(rec);
  const unsigned short* sl =
      reinterpret_cast<const unsigned short*>(rec + record_values(n, k, sizeof(T)));
  for (int j = 0; j < len; ++j) {
    int back = last % w - (int)sl[(j / 4 * n + lane) * 4 + j % 4];
    if (back < 0) back += w;
    if (rcol) rcol[s + j] = last - back;
    if (rval) rval[s + j] = v[((j + 1) / 2 * n + lane) * 2 + (j + 1) % 2];
  }
  if (rcol) rcol[s + len] = p;
  if (rval) rval[s + len] = v[2 * lane];
}

// ------------------------------------------------------------ solving

template <typename T>
__global__ void gather_by_perm(const T* __restrict__ b, const int* __restrict__ perm, int N,
                               T* __restrict__ out) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < N) out[p] = b[perm[p]];
}

// One factor to solve: yw holds b in level order and receives the solution.
template <typename T>
struct View {
  const int4* groups;
  const char* records;
  T* yw;
  int ngroups;
  int window;
  int kmax;
  int per_level;  // arrivals that close a level
};

template <typename T>
__global__ void scatter_by_perm(const T* __restrict__ yw, const int* __restrict__ perm, int N,
                                T* __restrict__ y) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < N) y[perm[p]] = yw[p];
}

// Wait for the phase of parity `parity`, bounded by ~2^31 cycles or by another
// wait's timeout, which is recorded; false then, and the caller's warp ends its
// work without a further arrival (one would count for a wrong phase).
__device__ __forceinline__ bool wait_phase(uint64_t* bar, uint32_t parity, int* status) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  int spins = 0;
  while (!mbar_try_wait(bar, parity)) {
    if ((++spins & 63) == 0 && (clock64() - t0 > (1LL << 31) || *(volatile const int*)status)) {
      atomicExch(status, SB_DEV_TIMEOUT_DEP);
      return false;
    }
  }
  return true;
}
__device__ __forceinline__ void arrive_count(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(count)
               : "memory");
}

template <typename T> struct pair_of;
template <> struct pair_of<float> { using V = float2; };
template <> struct pair_of<double> { using V = double2; };

// A group's rows in registers, one per lane: KU values (the diagonal first)
// and KU slots.  Absent entries read the ring's extra slot, which holds +0,
// with value +0: t never is -0 (it starts at +0), so adding +0 changes nothing.
// Lanes past the group's rows repeat its last row and store nothing.
template <typename T, int KU>
struct Rows {
  typename pair_of<T>::V v[KU / 2];
  uint2 s[KU / 4];
  T b;
};

template <typename T, int KU>
__device__ __forceinline__ void load_rows(Rows<T, KU>& r, const View<T>& f, int4 g, int lane) {
  using V = typename pair_of<T>::V;
  const int n = group_rows(g), k = group_len(g), l = min(lane, n - 1);
  const char* rec = f.records + 16LL * g.y;
  const V* v = reinterpret_cast<const V*>(rec) + l;
  const uint2* s = reinterpret_cast<const uint2*>(rec + record_values(n, k, sizeof(T))) + l;
  r.b = __ldcg(f.yw + g.x + l);
  if (record_pairs(k) == KU / 2) {
#pragma unroll
    for (int p = 0; p < KU / 2; ++p) r.v[p] = __ldg(v + p * n);
#pragma unroll
    for (int q = 0; q < KU / 4; ++q) r.s[q] = __ldg(s + q * n);
  } else {
    const unsigned none = (unsigned)f.window * 0x10001u;
#pragma unroll
    for (int p = 0; p < KU / 2; ++p) {
      r.v[p].x = r.v[p].y = T(0);
      if (p < record_pairs(k)) r.v[p] = __ldg(v + p * n);
    }
#pragma unroll
    for (int q = 0; q < KU / 4; ++q) {
      r.s[q] = make_uint2(none, none);
      if (q < record_quads(k)) r.s[q] = __ldg(s + q * n);
    }
  }
}

// Keeps the compiler from moving the computation of v behind a later wait.
__device__ __forceinline__ void pin(uint32_t& v) { asm volatile("" : "+r"(v)); }

__device__ __forceinline__ void ld_ring(float& v, uint32_t a) {
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
}
__device__ __forceinline__ void ld_ring(double& v, uint32_t a) {
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
}

// All rows of one factor by a block of NW warps: warp w takes groups w,
// w + NW, ...  A group's record is read one group ahead, and everything that
// does not depend on the values waited for is computed ahead of the wait for
// the level before, so that only the ring reads and the arithmetic follow it.  Level l is closed by the
// barrier done[l % kLevelBars], whose phase takes `per_level` arrivals: one
// for each of the level's groups, and those that the level has fewer with its
// first group's.  A warp waits for a level at most NW levels after the one it
// worked on last (its groups lie NW apart), so with kLevelBars >= 2 NW
// barriers the phase it waits for is the barrier's current one.
template <typename T, typename A, int KU, int NW>
__device__ __forceinline__ void solve_rows(const View<T>& f, T* ring, uint64_t* done, int* status) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int mine = f.ngroups > warp ? (f.ngroups - warp + NW - 1) / NW : 0;
  if (mine == 0) return;
  const int4* gp = f.groups + warp;
  int4 g0 = __ldg(gp), g1 = g0, g2 = g0;
  if (1 < mine) g1 = __ldg(gp + NW);
  Rows<T, KU> cur, nxt;
  load_rows(cur, f, g0, lane);
  int slot0 = g0.x % f.window;  // ring slot of the group's first row
  const uint32_t ring_a = smem_u32(ring);
  for (int it = 0; it < mine; ++it) {
    if (it + 1 < mine) load_rows(nxt, f, g1, lane);
    if (it + 2 < mine) g2 = __ldg(gp + (long long)(it + 2) * NW);
    uint32_t a[KU];
#pragma unroll
    for (int q = 0; q < KU / 4; ++q) {
      a[4 * q] = ring_a + (cur.s[q].x & 0xffffu) * (uint32_t)sizeof(T);
      a[4 * q + 1] = ring_a + (cur.s[q].x >> 16) * (uint32_t)sizeof(T);
      a[4 * q + 2] = ring_a + (cur.s[q].y & 0xffffu) * (uint32_t)sizeof(T);
      a[4 * q + 3] = ring_a + (cur.s[q].y >> 16) * (uint32_t)sizeof(T);
    }
#pragma unroll
    for (int j = 0; j < KU - 1; ++j) pin(a[j]);
    bool open = true;
    if (g0.z > 0)
      open = wait_phase(done + (g0.z - 1) % kLevelBars, ((g0.z - 1) / kLevelBars) & 1, status);
    T y[KU];
#pragma unroll
    for (int j = 0; j < KU - 1; ++j) ld_ring(y[j], a[j]);
    A t = 0;
#pragma unroll
    for (int j = 0; j < KU - 1; ++j) {
      const T v = (j + 1) % 2 ? cur.v[(j + 1) / 2].y : cur.v[(j + 1) / 2].x;
      t = add_rn(t, mul_rn((A)v, (A)y[j]));
    }
    const T yi = (T)div_rn(sub_rn((A)cur.b, t), (A)cur.v[0].x);
    const bool on = lane < group_rows(g0);
    const int slot = slot0 + lane < f.window ? slot0 + lane : slot0 + lane - f.window;
    if (on) ring[slot] = yi;
    if (!__all_sync(0xffffffffu, open)) return;
    __syncwarp();  // the lanes' ring stores before lane 0's arrival (a vote orders no memory)
    if (lane == 0) arrive_count(done + g0.z % kLevelBars, group_arrivals(g0));
    if (on) __stcg(f.yw + g0.x + lane, yi);
    slot0 += g1.x - g0.x;
    while (slot0 >= f.window) slot0 -= f.window;
    g0 = g1;
    g1 = g2;
    cur = nxt;
  }
}

// Warps of the block: as many as its registers allow, fewer where more
// measured slower (1M-row random factor, 7 entries a row, FP64: 1.68 ms with
// 16 warps, 1.76 with 24; FP32 1.33 and 1.18).
template <typename T, int KU> struct Warps {
  static constexpr int n = KU == 4 ? 32 : KU == 8 ? (sizeof(T) == 4 ? 24 : 16) : 12;
};

template <typename T, typename A, int KU>
__global__ void __launch_bounds__(32 * Warps<T, KU>::n, 1) window_solve(View<T> f, int* status) {
  extern __shared__ __align__(16) char smem[];
  __shared__ __align__(8) uint64_t done[kLevelBars];
  T* ring = reinterpret_cast<T*>(smem);
  if (threadIdx.x < kLevelBars) mbar_init(done + threadIdx.x, f.per_level);
  if (threadIdx.x == 0) ring[f.window] = T(0);
  mbar_fence_init();
  __syncthreads();
  solve_rows<T, A, KU, Warps<T, KU>::n>(f, ring, done, status);
}

// Several factors, one per block (the longest first).  KU: the largest of the
// batch.
template <typename T, typename A, int KU>
__global__ void __launch_bounds__(32 * Warps<T, KU>::n, 1)
    window_solve_many(const View<T>* __restrict__ views, const int* __restrict__ count,
                      int* status) {
  constexpr int NW = Warps<T, KU>::n;
  extern __shared__ __align__(16) char smem[];
  __shared__ __align__(8) uint64_t done[kLevelBars];
  T* ring = reinterpret_cast<T*>(smem);
  if ((int)blockIdx.x >= *count) return;
  const View<T> f = views[blockIdx.x];
  if (threadIdx.x < kLevelBars) mbar_init(done + threadIdx.x, f.per_level);
  if (threadIdx.x == 0) ring[f.window] = T(0);
  mbar_fence_init();
  __syncthreads();
  const int u = unroll_of(f.kmax);
  if (u == 4) solve_rows<T, A, 4, NW>(f, ring, done, status);
  if constexpr (KU >= 8)
    if (u == 8) solve_rows<T, A, 8, NW>(f, ring, done, status);
  if constexpr (KU >= 16)
    if (u == 16) solve_rows<T, A, 16, NW>(f, ring, done, status);
}

// b of every item into level order (SCATTER: the solutions back into natural
// order): one block per kMoveRows rows of an item; first[k] is item k's first
// block.
constexpr int kMoveRows = 1024;

template <typename T>
struct Move {
  const int* perm;
  const T* b;
  T* yw;
  T* y;
  int N;
  int first;
};

template <typename T, bool SCATTER>
__global__ void __launch_bounds__(256)
    window_move(const Move<T>* __restrict__ moves, const int* __restrict__ count) {
  int lo = 0, hi = *count - 1;  // the last item that starts at or before this block
  if (hi < 0) return;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (moves[mid].first <= (int)blockIdx.x) lo = mid;
    else hi = mid - 1;
  }
  const Move<T> m = moves[lo];
  const long long p0 = (long long)((int)blockIdx.x - m.first) * kMoveRows + threadIdx.x;
#pragma unroll
  for (int u = 0; u < kMoveRows / 256; ++u) {
    const long long p = p0 + u * 256;
    if (p < m.N) {
      const int i = __ldg(m.perm + p);
      if (SCATTER) m.y[i] = m.yw[p];
      else m.yw[p] = m.b[i];
    }
  }
}

}  // namespace
}  // namespace win
}  // namespace sb
