// sb_convert.cu -- format conversions on the device, bit-exact with the
// reference's JavaScript loops:
//   coo_csr   src/sequential/src/sparse32.js:1674-1720 (+ sort :1612-1627)
//   num_cols  :1436-1447 and csr_ell :1449-1484
//   num_diags :1486-1512 and csr_dia :1515-1574
// coo_csr's per-row stable bubble sort makes the result a stable sort of the
// COO entries by (row, col).  Sorted input (the reference's mmread always
// quick-sorts by (row, col)) is detected and takes a copy-speed path; other
// input goes through buckets of rows (sb_buckets.cu) unless a row is too long
// for them, and is otherwise ordered by a stable LSD radix sort of packed
// (row, col) keys whose payload is the original position; either way equal keys
// keep their COO order.
#include <algorithm>

#include <climits>

#include "sb_buckets.cuh"
#include "sb_prims.cuh"

namespace sb {

constexpr int kThreads = 256;

static unsigned grid_for(long long n, int per = kThreads) {
  long long g = (n + per - 1) / per;
  if (g < 1) g = 1;
  if (g > 0x7fffffffLL) g = 0x7fffffffLL;
  return (unsigned)g;
}

// flags[0] |= 1: index out of range; flags[1] |= 1: not sorted by (row, col).
// Each thread checks kCheckItems entries (strided by the block size, so every
// load is coalesced) and a block stores its findings once, and only while the
// flag still reads 0: in a shuffled COO nearly every entry is out of order,
// and one store per entry to the same word serialised (0.79 ms for 44M
// entries).
constexpr int kCheckItems = 8;

__global__ void coo_check(const int* __restrict__ row, const int* __restrict__ col, long long nnz,
                          int N, int* __restrict__ flags) {
  const long long base = (long long)blockIdx.x * blockDim.x * kCheckItems + threadIdx.x;
  int bad = 0, unsorted = 0;
#pragma unroll
  for (int u = 0; u < kCheckItems; ++u) {
    const long long i = base + (long long)u * blockDim.x;
    if (i < nnz) {
      const int r = row[i], c = col[i];
      bad |= (r < 0 || r >= N || c < 0 || c >= N);
      if (i + 1 < nnz) {
        const int r1 = row[i + 1], c1 = col[i + 1];
        unsorted |= (r1 < r || (r1 == r && c1 < c));
      }
    }
  }
  bad = __syncthreads_or(bad);
  unsorted = __syncthreads_or(unsorted);
  if (threadIdx.x == 0) {
    if (bad && __ldcg(flags) == 0) flags[0] = 1;
    if (unsorted && __ldcg(flags + 1) == 0) flags[1] = 1;
  }
}

__global__ void pack_keys(const int* __restrict__ row, const int* __restrict__ col,
                          long long nnz, unsigned long long* __restrict__ keys,
                          unsigned* __restrict__ idx) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nnz) return;
  keys[i] = ((unsigned long long)(unsigned)row[i] << 32) | (unsigned)col[i];
  idx[i] = (unsigned)i;
}

template <typename T>
__global__ void unpack_sorted(const unsigned long long* __restrict__ keys,
                              const unsigned* __restrict__ idx, const T* __restrict__ val,
                              long long nnz, int* __restrict__ row_out, int* __restrict__ col_out,
                              T* __restrict__ val_out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nnz) return;
  const unsigned long long k = keys[i];
  row_out[i] = (int)(k >> 32);
  col_out[i] = (int)(k & 0xffffffffu);
  val_out[i] = val[idx[i]];
}

// max row length (num_cols)
__global__ void max_row_len(const int* __restrict__ row_ptr, int N, int* __restrict__ out) {
  __shared__ int sm[32];
  int m = 0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < N;
       i += (long long)gridDim.x * blockDim.x)
    m = max(m, row_ptr[i + 1] - row_ptr[i]);
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x < 32) {
    m = threadIdx.x < (blockDim.x >> 5) ? sm[threadIdx.x] : 0;
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (threadIdx.x == 0) atomicMax(out, m);
  }
}

// csr_ell: thread per row writes all nc slots of its row (entries in storage
// order, then zero padding with index 0), column-major slot k*N + i.
template <typename T>
__global__ void csr_to_ell(const int* __restrict__ row_ptr, const int* __restrict__ col,
                           const T* __restrict__ val, int N, int nc, int* __restrict__ indices,
                           T* __restrict__ data) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const int s = row_ptr[i], e = row_ptr[i + 1];
  for (int k = 0; k < nc; ++k) {
    const long long o = (long long)k * N + i;
    const int j = s + k;
    if (j < e) {
      indices[o] = col[j];
      data[o] = val[j];
    } else {
      indices[o] = 0;
      data[o] = (T)0;
    }
  }
}

// The diagonals c - i (c a column within the matrix, i its row) that occur.
// A stencil's or a band's matrix has few, and its first and last rows show
// them all: `known_diagonals` collects those of the first and last 512 rows
// in a hash table, and where they are at most kDiaGather the other rows are
// only held against that list.  A diagonal outside it (a stray), or a matrix
// of many, is marked in one byte per diagonal, at N + c - i - 1 as in the
// reference (:1498), and the bytes are counted and ranked by tiles.
// A 4M-row band of 11 diagonals on B200, num_diags: one 4-byte flag per
// diagonal, stored by every row and scanned, 115 us of device time; now 57,
// 47 of them in mark_diagonals (29 at copy speed for the columns).  csr_dia,
// which needed the same once more, finds the list in 8 us and checks the
// entries in its fill.
constexpr int kDiaGather = 64;
constexpr int kKnownRows = 512;  // at each end

struct Known {
  int count;  // of the first and last rows; kDiaGather + 1: more
  int stray;  // set: a row has a diagonal outside offset[0 .. count)
  int check;  // set: a diagonal's byte is read before it is stored (mark_all)
  int offset[kDiaGather];
};

constexpr int kSlots = 256;

__device__ __forceinline__ void insert_offset(int d, int* key, int* count) {
  unsigned h = ((unsigned)d * 2654435761u) >> 24;
  for (int step = 0; step < kSlots && *(volatile int*)count <= kDiaGather;
       ++step, h = (h + 1) & (kSlots - 1)) {
    int at = *(volatile int*)&key[h];
    if (at == INT_MAX) {
      at = atomicCAS(&key[h], INT_MAX, d);
      if (at == INT_MAX) {
        atomicAdd(count, 1);
        return;
      }
    }
    if (at == d) return;
  }
}

// present (zero on entry; may be null): where there are too many for the list, the
// diagonals of a few rows are marked ahead of all others, so that the warps
// of mark_all that start together find the bytes of a wide stencil set instead of
// all storing to the same few sectors; and they tell whether rows share their
// diagonals at all.
constexpr int kSeedRows = 8;        // of the middle
constexpr int kSeedEntries = 1024;  // of a row at most

__global__ void __launch_bounds__(2 * kKnownRows)
    known_diagonals(const int* __restrict__ row_ptr, const int* __restrict__ col, int N,
                    Known* __restrict__ known, unsigned char* __restrict__ present) {
  __shared__ int key[kSlots];
  __shared__ int count;
  const int t = threadIdx.x;
  if (t < kSlots) key[t] = INT_MAX;  // (no diagonal: c - i < N)
  if (t == 0) count = 0;
  __syncthreads();
  const int i = t < kKnownRows ? t : N - 1 - (t - kKnownRows);
  int s = 0, e = 0;
  if (t < kKnownRows ? i < N : i >= kKnownRows) {
    s = row_ptr[i];
    e = row_ptr[i + 1];
  }
  if (e - s > kDiaGather) {
    atomicAdd(&count, kDiaGather + 1);
    e = s;
  }
  constexpr int kAhead = 8;
  for (int t0 = 0; t0 < e - s && *(volatile int*)&count <= kDiaGather; t0 += kAhead) {
    int c[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) c[u] = t0 + u < e - s ? col[s + t0 + u] : -1;
#pragma unroll 1
    for (int u = 0; u < kAhead; ++u) {
      if ((unsigned)c[0] < (unsigned)N) insert_offset(c[0] - i, key, &count);
#pragma unroll
      for (int v = 0; v + 1 < kAhead; ++v) c[v] = c[v + 1];
    }
  }
  __syncthreads();
  const int n = min(count, kDiaGather + 1);
  if (t == 0) {
    known->count = n;
    known->stray = 0;
  }
  if (n <= kDiaGather && t < kSlots && key[t] != INT_MAX) {
    int rank = 0;
    for (int k = 0; k < kSlots; ++k) rank += key[k] < key[t];
    known->offset[rank] = key[t];
  }
  if (n > kDiaGather && present) {
    // one warp to a row: four from the middle, the first and the last four (where
    // one-sided diagonals begin), then the next four of the middle, held against
    // what the others marked
    __shared__ int seen, all;
    if (t == 0) seen = all = 0;
    __syncthreads();
    const int w = t >> 5;
    const int r = w < kSeedRows ? N / 2 + w : w < 12 ? w - kSeedRows : N - 1 - (w - 12);
    const bool mine = w < 16 && r >= 0 && r < N;
    const int s0 = mine ? row_ptr[r] : 0, len = mine ? min(row_ptr[r + 1] - s0, kSeedEntries) : 0;
    for (int half = 0; half < 2; ++half) {
      if ((w >= 4 && w < kSeedRows) == (half == 1))
        for (int j = t & 31; j < len; j += 32) {
          const int c = col[s0 + j];
          if ((unsigned)c >= (unsigned)N) continue;
          unsigned char* f = present + ((long long)N + c - r - 1);
          if (half) {
            atomicAdd(&all, 1);
            if (*(volatile unsigned char*)f) atomicAdd(&seen, 1);
          }
          *f = 1;
        }
      __syncthreads();
    }
    if (t == 0) known->check = 2 * seen > all;
  }
}

// The first of n ascending offsets that is not below d.
__device__ __forceinline__ int first_place(long long d, const int* off, int n) {
  int k = 0;
  while (k < n && off[k] < d) ++k;
  return k;
}

// Whether a row's entries (one at least) lie on consecutive offsets, as almost
// every row of a band or a stencil does.  The loads don't wait on one another.
__device__ __forceinline__ bool run_of_offsets(const int* __restrict__ col, int s, int e, int i,
                                               int N, const int* off, int n) {
  const int k0 = first_place(col[s] - (long long)i, off, n);
  if (e - s > n - k0) return false;
  bool ok = true;
#pragma unroll 8
  for (int u = 0; u < e - s; ++u) {
    const int c = col[s + u];
    ok &= (unsigned)c < (unsigned)N && c - i == off[k0 + u];
  }
  return ok;
}

// Every diagonal of the rows into present: a warp takes `rows` (at most 32)
// rows at a time and its lanes their entries in storage order, so that loads
// coalesce and long rows are shared out; an entry's row is found among the
// row pointers.  A byte is stored only while it reads 0 (a stale 0 costs one
// more idempotent store) where rows share their diagonals (known->check) or 32
// entries in a row lie on near ones, as the same few sectors would otherwise be
// stored over and over; elsewhere the check would be a round trip for nothing.
// num_diags on B200, the whole call in us (4-byte flags and a thread per row /
// bytes checked on near diagonals alone / now): 30,000 rows of 80 diagonals 97 /
// 77-130 / 58, 300,000 rows 307 / 134 / 121; 100 diagonals 97 apart, 300,000 rows
// 187 / 8960 / 143; 125-point stencil of 1.5M rows 757 / 5025 / 563; power law of 2M
// rows 529 / 430 / 430.  Random columns lose what the bytes save on structure: 60
// entries a row, 300,000 rows 222 / 290 / 290 (checked 315), 10,000 rows 88 / 178 /
// 178 (checked 253).
constexpr int kNarrow = 4096;

__device__ void mark_all(const int* __restrict__ row_ptr, const int* __restrict__ col, int N,
                         int rows, bool always, int (*ptr)[33], unsigned char* present) {
  const int lane = threadIdx.x & 31;
  int* p = ptr[threadIdx.x >> 5];
  const int warps = gridDim.x * (kThreads / 32);
  const int chunks = (N - 1) / rows + 1;
  for (int q = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5); q < chunks; q += warps) {
    const int r0 = q * rows, n = min(rows, N - r0);
    p[lane] = row_ptr[r0 + min(lane, n)];
    if (lane == 0) p[32] = row_ptr[r0 + n];
    __syncwarp();
    const int s = p[0], e = p[32];
    if (__any_sync(0xffffffffu, p[lane] > p[lane + 1])) {  // row pointers that don't ascend
      if (lane < n)
        for (int j = p[lane], end = row_ptr[r0 + lane + 1]; j < end; ++j) {
          const int c = col[j];
          if ((unsigned)c < (unsigned)N) present[(long long)N + c - (r0 + lane) - 1] = 1;
        }
      __syncwarp();
      continue;
    }
    constexpr int kAhead = 4;
    const unsigned len = (unsigned)e - (unsigned)s;
    for (unsigned t0 = 0; t0 < len; t0 += 32 * kAhead) {
      const unsigned t = t0 + lane;
      int c[kAhead];
      long long at[kAhead];  // the byte to set, < 0: none
      unsigned char have[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) c[u] = t + 32 * u < len ? col[s + t + 32 * u] : -1;
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        int r = 0;  // the last row that begins at or before the entry
#pragma unroll
        for (int step = 16; step > 0; step >>= 1)
          if ((unsigned)p[r + step] - (unsigned)s <= t + 32 * u) r += step;
        at[u] = (unsigned)c[u] < (unsigned)N ? (long long)N + c[u] - (r0 + r) - 1 : -1;
      }
      const unsigned lo = __reduce_min_sync(0xffffffffu, at[0] >= 0 ? (unsigned)at[0] : ~0u);
      const unsigned hi = __reduce_max_sync(0xffffffffu, at[0] >= 0 ? (unsigned)at[0] : 0u);
      const bool check = always || hi - lo < (unsigned)kNarrow;
#pragma unroll
      for (int u = 0; u < kAhead; ++u)
        have[u] = at[u] >= 0 ? (check ? present[at[u]] : (unsigned char)0) : (unsigned char)1;
#pragma unroll
      for (int u = 0; u < kAhead; ++u)
        if (!have[u]) present[at[u]] = 1;
    }
    __syncwarp();
  }
}

// present is zero on entry.
__global__ void __launch_bounds__(kThreads)
    mark_diagonals(const int* __restrict__ row_ptr, const int* __restrict__ col, int N, int rows,
                   Known* __restrict__ known, unsigned char* __restrict__ present) {
  __shared__ int off[kDiaGather];
  __shared__ int ptr[kThreads / 32][33];
  const int n = known->count;
  if (n > kDiaGather) {
    mark_all(row_ptr, col, N, rows, known->check, ptr, present);
    return;
  }
  if (threadIdx.x < n) {
    off[threadIdx.x] = known->offset[threadIdx.x];
    if (blockIdx.x == 0) present[(long long)N + off[threadIdx.x] - 1] = 1;
  }
  __syncthreads();
  bool stray = false;
  for (long long r = (long long)blockIdx.x * kThreads + threadIdx.x; r < N;
       r += (long long)gridDim.x * kThreads) {
    const int i = (int)r, s = row_ptr[i], e = row_ptr[i + 1];
    if (s >= e || run_of_offsets(col, s, e, i, N, off, n)) continue;
    for (int j = s; j < e; ++j) {
      const int c = col[j];
      if ((unsigned)c >= (unsigned)N) continue;
      const int k = first_place(c - i, off, n);
      if (k < n && off[k] == c - i) continue;
      unsigned char* f = present + ((long long)N + c - i - 1);
      if (*f == 0) *f = 1;
      stray = true;
    }
  }
  if (__syncthreads_or(stray) && threadIdx.x == 0) known->stray = 1;
}

// Counts per tile of 16 bytes a thread, and from the scanned counts the
// present diagonals' offsets in ascending order and (where asked for) ranks.
__device__ __forceinline__ int ones(uint4 b) {  // bytes of 0 or 1
  return __popc(b.x) + __popc(b.y) + __popc(b.z) + __popc(b.w);
}

__global__ void __launch_bounds__(kThreads)
    count_bytes(const uint4* __restrict__ present, long long words, int* __restrict__ sums) {
  const long long w = (long long)blockIdx.x * kThreads + threadIdx.x;
  __shared__ int total;
  if (threadIdx.x == 0) total = 0;
  __syncthreads();
  const int c = __reduce_add_sync(0xffffffffu, w < words ? ones(present[w]) : 0);
  if ((threadIdx.x & 31) == 0) atomicAdd(&total, c);
  __syncthreads();
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kThreads)
    compact_diagonals(const uint4* __restrict__ present, long long words,
                      const int* __restrict__ start, int N, int* __restrict__ offset,
                      int* __restrict__ rank) {
  __shared__ int warp_sum[kThreads / 32];
  const long long w = (long long)blockIdx.x * kThreads + threadIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint4 b = w < words ? present[w] : make_uint4(0, 0, 0, 0);
  const int mine = ones(b);
  int incl = mine;
  for (int o = 1; o < 32; o <<= 1) {
    const int up = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += up;
  }
  if (lane == 31) warp_sum[warp] = incl;
  __syncthreads();
  if (mine == 0) return;
  int at = start[blockIdx.x] + incl - mine;
  for (int k = 0; k < warp; ++k) at += warp_sum[k];
  const unsigned q[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    if ((q[k >> 2] >> (8 * (k & 3)) & 1u) == 0) continue;
    const long long d = w * 16 + k;
    offset[at] = (int)(d - (N - 1));
    if (rank) rank[d] = at;
    ++at;
  }
}

// csr_dia fill for at most kDiaGather diagonals: thread per row; slot k of
// row i receives the row's LAST entry in column i + offset[k] (the
// reference's row-major loop, :1559-1571, lets a later duplicate overwrite
// an earlier one), else +0, so every slot is written with writes coalesced
// across rows, and no zero fill or scatter is needed.  A row is taken as a
// run of consecutive offsets, its loads independent of one another; where
// that proves wrong its slots are written again by a search per slot.  Loads
// go in batches of 5 slots (batches of 3 and 8 measured the same, 9 or a plain
// unrolled loop 9-30% longer).  Comparing 16 entries in registers with every
// slot took 211 us for a 4M-row FP64 band of 11 diagonals on B200; now 146, at
// 6.1 TB/s of row pointers, entries and slots.  Entries staged in shared
// memory measured longer (195).  CHECK: an entry outside the offsets is
// reported.
template <typename T, bool CHECK>
__global__ void __launch_bounds__(kThreads)
    csr_to_dia_rows(const int* __restrict__ row_ptr, const int* __restrict__ col,
                    const T* __restrict__ val, int N, int nd, const int* __restrict__ offset,
                    T* __restrict__ data, int* __restrict__ stray) {
  __shared__ int off[kDiaGather];
  const int i = blockIdx.x * kThreads + threadIdx.x;
  if (threadIdx.x < nd) off[threadIdx.x] = offset[threadIdx.x];
  __syncthreads();
  if (i >= N) return;
  const int s = row_ptr[i], len = max(row_ptr[i + 1] - s, 0);
  const int k0 = len > 0 ? first_place(col[s] - (long long)i, off, nd) : 0;
  bool ok = len <= nd - k0;
  constexpr int kAhead = 5;
  for (int kb = 0; kb < nd; kb += kAhead) {
    int c[kAhead];
    T v[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int j = kb + u - k0;
      const bool in = (unsigned)j < (unsigned)len && kb + u < nd;
      c[u] = in ? col[s + j] : i + off[min(kb + u, nd - 1)];
      v[u] = in ? val[s + j] : T(0);
      ok &= !in || (unsigned)c[u] < (unsigned)N;
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
      if (kb + u < nd) {
        ok &= c[u] - i == off[kb + u];
        data[(long long)(kb + u) * N + i] = v[u];
      }
  }
  if (ok) return;
  for (int k = 0; k < nd; ++k) {
    const int want = off[k];
    T out = T(0);
    for (int j = s; j < s + len; ++j) {
      const int c = col[j];
      // out-of-range columns are not stored (the reference skips them)
      if ((unsigned)c < (unsigned)N && c - i == want) out = val[j];
    }
    data[(long long)k * N + i] = out;
  }
  for (int j = s; CHECK && j < s + len; ++j) {
    const int c = col[j];
    if ((unsigned)c >= (unsigned)N) continue;
    const int k = first_place(c - i, off, nd);
    if (k == nd || off[k] != c - i) *stray = 1;
  }
}

// csr_dia fill: thread per row, entries in storage order so a later
// duplicate (i, c) overwrites an earlier one exactly as the reference's
// row-major loop does (:1559-1571).  data is zero-filled beforehand.
template <typename T>
__global__ void csr_to_dia(const int* __restrict__ row_ptr, const int* __restrict__ col,
                           const T* __restrict__ val, int N, int stride,
                           const int* __restrict__ rank, T* __restrict__ data) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const long long move = (long long)N - stride;
  for (int j = row_ptr[i]; j < row_ptr[i + 1]; ++j) {
    const int c = col[j];
    if (c < 0 || c >= N) continue;
    const int k = rank[(long long)N + c - i - 1];
    const long long o = (long long)k * stride + i - ((c - i) < 0 ? move : 0);
    data[o] = val[j];
  }
}

static int check_dt(int dtype, const char* fn) {
  if (dtype != SB_F32 && dtype != SB_F64) {
    set_error("%s: dtype %d not supported", fn, dtype);
    return SB_EINVAL;
  }
  return SB_OK;
}

// Host-side admission test of csr_ell / csr_dia, evaluated in doubles as in
// JavaScript: admit iff w*N < 2^27 and (w*N)/nnz <= 5 (0/0 is NaN: refused).
static bool admitted(long long w, long long N, long long nnz) {
  const double wn = (double)w * (double)N;
  const double ratio = wn / (double)nnz;
  return (wn < 134217728.0) && (ratio <= 5.0);
}

constexpr int kCheckPrefix = 1 << 16;

// coo_check's flags for the first n entries, on the host.
static int check_order(const int* row, const int* col, long long n, int N, int (&hf)[2],
                       cudaStream_t st) {
  int* flags = nullptr;
  const int r = scratch_alloc((void**)&flags, 2 * sizeof(int), st);
  if (r) return r;
  SB_CHECK_CUDA(cudaMemsetAsync(flags, 0, 2 * sizeof(int), st));
  coo_check<<<grid_for(n, kThreads * kCheckItems), kThreads, 0, st>>>(row, col, n, N, flags);
  SB_CHECK_LAUNCH("coo_check");
  SB_CHECK_CUDA(cudaMemcpyAsync(hf, flags, sizeof(hf), cudaMemcpyDeviceToHost, st));
  SB_CHECK_CUDA(cudaStreamSynchronize(st));
  scratch_free(flags, st);
  return SB_OK;
}

template <typename T>
static int coo_csr_impl(const int* row, const int* col, const T* val, int N, long long nnz,
                        int* csr_row, int* csr_col, T* csr_val, cudaStream_t st) {
  // the order of a prefix first: shuffled entries show there, and then their
  // indices are checked by the pass that counts them
  int hf[2] = {0, 0};
  long long checked = std::min(nnz, (long long)kCheckPrefix);
  int r = check_order(row, col, checked, N, hf, st);
  if (!r && !hf[0] && !hf[1] && checked < nnz) {
    checked = nnz;
    r = check_order(row, col, nnz, N, hf, st);
  }
  if (r) return r;
  if (hf[0]) {
    set_error("coo_csr: row or column index outside [0, N)");
    return SB_EINVAL;
  }
  if (!hf[1]) {
    // already in (row, col) order: the stable sort is the identity
    SB_CHECK_CUDA(cudaMemcpyAsync(csr_col, col, sizeof(int) * nnz, cudaMemcpyDeviceToDevice, st));
    SB_CHECK_CUDA(cudaMemcpyAsync(csr_val, val, sizeof(T) * nnz, cudaMemcpyDeviceToDevice, st));
    prim::row_ptr_from_sorted<<<grid_for(nnz + 1), kThreads, 0, st>>>(row, nnz, N, csr_row);
    SB_CHECK_LAUNCH("row_ptr_from_sorted");
    return SB_OK;
  }
  // any order: buckets of rows
  r = bucket_csr<T>(row, col, nullptr, val, N, N, nnz, checked < nnz, csr_row, csr_col,
                    csr_val, st);
  if (r != kBucketsUnfit) return r;
  // rows beyond a bucket: stable radix sort of (row << 32 | col) with positions
  prim::RadixBuffers b;
  void* mem = nullptr;
  const size_t kb = sizeof(unsigned long long) * (size_t)nnz, vb = sizeof(unsigned) * (size_t)nnz;
  r = scratch_alloc(&mem, 2 * kb + 2 * vb + sizeof(int) * (size_t)nnz, st);
  if (r) return r;
  char* p = (char*)mem;
  b.k[0] = (unsigned long long*)p;
  b.k[1] = (unsigned long long*)(p + kb);
  b.v[0] = (unsigned*)(p + 2 * kb);
  b.v[1] = (unsigned*)(p + 2 * kb + vb);
  int* rows_sorted = (int*)(p + 2 * kb + 2 * vb);
  pack_keys<<<grid_for(nnz), kThreads, 0, st>>>(row, col, nnz, b.k[0], b.v[0]);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) r = cuda_status(e, "pack_keys");
  const int nb = prim::bits_for(N > 0 ? N - 1 : 0);
  const int ranges[4] = {0, nb, 32, 32 + nb};
  int which = 0;
  if (!r) r = prim::radix_sort_ranges(b, nnz, ranges, 2, &which, st);
  if (!r) {
    unpack_sorted<T><<<grid_for(nnz), kThreads, 0, st>>>(b.k[which], b.v[which], val, nnz,
                                                         rows_sorted, csr_col, csr_val);
    e = cudaGetLastError();
    if (e != cudaSuccess) r = cuda_status(e, "unpack_sorted");
  }
  if (!r) {
    prim::row_ptr_from_sorted<<<grid_for(nnz + 1), kThreads, 0, st>>>(rows_sorted, nnz, N, csr_row);
    e = cudaGetLastError();
    if (e != cudaSuccess) r = cuda_status(e, "row_ptr_from_sorted");
  }
  if (!r) {
    e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) r = cuda_status(e, "coo_csr");
  }
  scratch_free(mem, st);
  return r;
}

// Presence bytes (a whole number of uint4) and the starts of their tiles, with
// the total after them.
struct Diags {
  long long words, tiles;
  uint4* present;
  int* start;
  Known* known;
  char* mem;
};

static int diags_alloc(int N, Diags& d, cudaStream_t st) {
  d.words = (2LL * N - 1 + 15) / 16;
  d.tiles = (d.words + kThreads - 1) / kThreads;
  const size_t kb = (sizeof(Known) + 15) & ~(size_t)15;
  const int r = scratch_alloc((void**)&d.mem, sizeof(uint4) * (size_t)d.words + kb +
                                                  sizeof(int) * (size_t)(d.tiles + 1), st);
  if (r) return r;
  d.present = reinterpret_cast<uint4*>(d.mem);
  d.known = reinterpret_cast<Known*>(d.present + d.words);
  d.start = reinterpret_cast<int*>(reinterpret_cast<char*>(d.known) + kb);
  return SB_OK;
}

// The number of diagonals into *nd; all: also the presence bytes and tile
// starts (left out where the first and last rows show every diagonal).
static int find_diagonals(const int* row_ptr, const int* col, int N, const Diags& d, bool all,
                          int* nd, cudaStream_t st) {
  unsigned char* present = reinterpret_cast<unsigned char*>(d.present);
  SB_CHECK_CUDA(cudaMemsetAsync(present, 0, sizeof(uint4) * (size_t)d.words, st));
  known_diagonals<<<1, 2 * kKnownRows, 0, st>>>(row_ptr, col, N, d.known, present);
  const unsigned grid = (unsigned)sm_count() * 8;
  // rows a warp of mark_all takes: as many as leave every warp some, 1 to 32
  int rows = 32;
  while (rows > 1 && (long long)rows * grid * (kThreads / 32) > N) rows >>= 1;
  mark_diagonals<<<grid, kThreads, 0, st>>>(row_ptr, col, N, rows, d.known, present);
  SB_CHECK_LAUNCH("mark_diagonals");
  int head[2] = {0, 0};  // known->count, known->stray
  SB_CHECK_CUDA(cudaMemcpyAsync(head, d.known, sizeof(head), cudaMemcpyDeviceToHost, st));
  SB_CHECK_CUDA(cudaStreamSynchronize(st));
  *nd = head[0];
  if (!all && head[0] <= kDiaGather && !head[1]) return SB_OK;
  SB_CHECK_CUDA(cudaMemsetAsync(d.start + d.tiles, 0, sizeof(int), st));
  count_bytes<<<(unsigned)d.tiles, kThreads, 0, st>>>(d.present, d.words, d.start);
  SB_CHECK_LAUNCH("count_bytes");
  const int r = prim::exclusive_scan(d.start, d.start, d.tiles + 1, st);
  if (r) return r;
  SB_CHECK_CUDA(cudaMemcpyAsync(nd, d.start + d.tiles, sizeof(int), cudaMemcpyDeviceToHost, st));
  SB_CHECK_CUDA(cudaStreamSynchronize(st));
  return SB_OK;
}

static int num_diags_impl(const int* row_ptr, const int* col, int N, int* nd, cudaStream_t st) {
  Diags d;
  int r = diags_alloc(N, d, st);
  if (r) return r;
  r = find_diagonals(row_ptr, col, N, d, false, nd, st);
  scratch_free(d.mem, st);
  return r;
}

// csr_dia of a matrix whose first and last rows show all of its nd diagonals:
// *done set once the arrays are complete.  The fill itself checks every entry.
template <typename T>
static int csr_dia_known(const int* row_ptr, const int* col, const T* val, int N, int nd,
                         int* offset, T* data, bool* done, cudaStream_t st) {
  *done = false;
  Known* known = nullptr;
  int r = scratch_alloc((void**)&known, sizeof(Known), st);
  if (r) return r;
  int head[2] = {0, 0};
  known_diagonals<<<1, 2 * kKnownRows, 0, st>>>(row_ptr, col, N, known, nullptr);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(head, known, sizeof(head), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e == cudaSuccess && head[0] == nd && nd <= kDiaGather) {
    e = cudaMemcpyAsync(offset, known->offset, sizeof(int) * (size_t)nd, cudaMemcpyDeviceToDevice,
                        st);
    if (e == cudaSuccess) {
      csr_to_dia_rows<T, true><<<grid_for(N), kThreads, 0, st>>>(row_ptr, col, val, N, nd,
                                                                known->offset, data, &known->stray);
      e = cudaGetLastError();
    }
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(head, known, sizeof(head), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    *done = e == cudaSuccess && !head[1];
  }
  scratch_free(known, st);
  return e == cudaSuccess ? SB_OK : cuda_status(e, "sb_csr_dia");
}

template <typename T>
static int csr_dia_impl(const int* row_ptr, const int* col, const T* val, int N, int nd,
                        int stride, int* offset, T* data, cudaStream_t st) {
  bool done = false;
  int r = csr_dia_known(row_ptr, col, val, N, nd, offset, data, &done, st);
  if (r || done) return r;
  Diags d;
  if ((r = diags_alloc(N, d, st))) return r;
  int* rank = nullptr;
  int nd_found = 0;
  r = find_diagonals(row_ptr, col, N, d, true, &nd_found, st);
  if (!r && nd_found != nd) {
    set_error("sb_csr_dia: nd=%d does not match the matrix (%d diagonals)", nd, nd_found);
    r = SB_EINVAL;
  }
  if (!r && nd > kDiaGather)
    r = scratch_alloc((void**)&rank, sizeof(int) * (size_t)(2LL * N - 1), st);
  if (!r) {
    compact_diagonals<<<(unsigned)d.tiles, kThreads, 0, st>>>(d.present, d.words, d.start, N,
                                                              offset, rank);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess && nd <= kDiaGather) {
      // gather: every slot written once (stride == N)
      csr_to_dia_rows<T, false><<<grid_for(N), kThreads, 0, st>>>(row_ptr, col, val, N, nd, offset,
                                                                 data, nullptr);
      e = cudaGetLastError();
    } else if (e == cudaSuccess) {
      e = cudaMemsetAsync(data, 0, sizeof(T) * (size_t)nd * (size_t)stride, st);
      if (e == cudaSuccess) {
        csr_to_dia<T><<<grid_for(N), kThreads, 0, st>>>(row_ptr, col, val, N, stride, rank, data);
        e = cudaGetLastError();
      }
    }
    if (e != cudaSuccess) r = cuda_status(e, "sb_csr_dia");
  }
  if (rank) scratch_free(rank, st);
  scratch_free(d.mem, st);
  return r;
}

}  // namespace sb

using namespace sb;

extern "C" {

int sb_coo_csr(int dtype, const int32_t* row, const int32_t* col, const void* val, int32_t N,
               int64_t nnz, int32_t* csr_row_ptr, int32_t* csr_col, void* csr_val,
               void* stream) {
  SB_TRACE("sb_coo_csr");
  int r = check_dt(dtype, "sb_coo_csr");
  if (r) return r;
  SB_REQUIRE(N >= 0 && nnz >= 0, "sb_coo_csr: negative size");
  SB_REQUIRE(nnz <= 0x7fffffffLL, "sb_coo_csr: nnz exceeds int32 row_ptr range");
  SB_REQUIRE(csr_row_ptr, "sb_coo_csr: null row_ptr");
  if ((r = ensure_device())) return r;
  cudaStream_t st = as_stream(stream);
  if (nnz == 0) {
    SB_CHECK_CUDA(cudaMemsetAsync(csr_row_ptr, 0, sizeof(int) * ((size_t)N + 1), st));
    SB_CHECK_CUDA(cudaStreamSynchronize(st));
    return SB_OK;
  }
  SB_REQUIRE(row && col && val && csr_col && csr_val, "sb_coo_csr: null pointer");
  if (dtype == SB_F32)
    return coo_csr_impl<float>(row, col, (const float*)val, N, nnz, csr_row_ptr, csr_col,
                               (float*)csr_val, st);
  return coo_csr_impl<double>(row, col, (const double*)val, N, nnz, csr_row_ptr, csr_col,
                              (double*)csr_val, st);
}

int sb_num_cols(const int32_t* row_ptr, int32_t N, int32_t* nc, void* stream) {
  SB_TRACE("sb_num_cols");
  SB_REQUIRE(nc && N >= 0, "sb_num_cols: bad argument");
  *nc = 0;
  if (N == 0) return SB_OK;
  SB_REQUIRE(row_ptr, "sb_num_cols: null row_ptr");
  int r = ensure_device();
  if (r) return r;
  cudaStream_t st = as_stream(stream);
  int* out = nullptr;
  if ((r = scratch_alloc((void**)&out, sizeof(int), st))) return r;
  SB_CHECK_CUDA(cudaMemsetAsync(out, 0, sizeof(int), st));
  const unsigned g = std::min<unsigned>(grid_for(N), (unsigned)sm_count() * 8);
  max_row_len<<<g, kThreads, 0, st>>>(row_ptr, N, out);
  SB_CHECK_LAUNCH("max_row_len");
  SB_CHECK_CUDA(cudaMemcpyAsync(nc, out, sizeof(int), cudaMemcpyDeviceToHost, st));
  SB_CHECK_CUDA(cudaStreamSynchronize(st));
  scratch_free(out, st);
  return SB_OK;
}

int sb_ell_admitted(int64_t ncols, int32_t N, int64_t nnz) {
  return admitted(ncols, N, nnz) ? 1 : 0;
}

int sb_csr_ell(int dtype, const int32_t* row_ptr, const int32_t* col, const void* val, int32_t N,
               int64_t nnz, int32_t nc, int32_t* indices, void* data, void* stream) {
  SB_TRACE("sb_csr_ell");
  int r = check_dt(dtype, "sb_csr_ell");
  if (r) return r;
  SB_REQUIRE(N >= 0 && nnz >= 0 && nc >= 0, "sb_csr_ell: negative size");
  if (!admitted(nc, N, nnz)) {
    set_error("csr_ell: not efficient to store this matrix in ELL (nc*N=%lld, nnz=%lld)",
              (long long)nc * N, (long long)nnz);
    return SB_EREFUSED;
  }
  SB_REQUIRE(row_ptr && indices && data && (nnz == 0 || (col && val)), "sb_csr_ell: null pointer");
  if ((r = ensure_device())) return r;
  cudaStream_t st = as_stream(stream);
  if (dtype == SB_F32)
    csr_to_ell<float><<<grid_for(N), kThreads, 0, st>>>(row_ptr, col, (const float*)val, N, nc,
                                                        indices, (float*)data);
  else
    csr_to_ell<double><<<grid_for(N), kThreads, 0, st>>>(row_ptr, col, (const double*)val, N, nc,
                                                         indices, (double*)data);
  SB_CHECK_LAUNCH("csr_to_ell");
  return SB_OK;
}

int sb_num_diags(const int32_t* row_ptr, const int32_t* col, int32_t N, int32_t* nd,
                 int32_t* stride, void* stream) {
  SB_TRACE("sb_num_diags");
  SB_REQUIRE(nd && stride && N >= 0, "sb_num_diags: bad argument");
  *nd = 0;
  *stride = N;
  if (N == 0) return SB_OK;
  SB_REQUIRE(row_ptr && col, "sb_num_diags: null pointer");
  int r = ensure_device();
  if (r) return r;
  cudaStream_t st = as_stream(stream);
  return num_diags_impl(row_ptr, col, N, nd, st);
}

int sb_dia_admitted(int64_t ndiags, int32_t stride, int64_t nnz) {
  return admitted(ndiags, stride, nnz) ? 1 : 0;
}

int sb_csr_dia(int dtype, const int32_t* row_ptr, const int32_t* col, const void* val, int32_t N,
               int64_t nnz, int32_t nd, int32_t stride, int32_t* offset, void* data,
               void* stream) {
  SB_TRACE("sb_csr_dia");
  int r = check_dt(dtype, "sb_csr_dia");
  if (r) return r;
  SB_REQUIRE(N >= 0 && nnz >= 0 && nd >= 0, "sb_csr_dia: negative size");
  SB_REQUIRE(stride == N, "sb_csr_dia: stride must equal N (reference :1510)");
  if (!admitted(nd, stride, nnz)) {
    set_error("csr_dia: not efficient to store this matrix in DIA (nd*stride=%lld, nnz=%lld)",
              (long long)nd * stride, (long long)nnz);
    return SB_EREFUSED;
  }
  SB_REQUIRE(row_ptr && col && val && offset && data, "sb_csr_dia: null pointer");
  if ((r = ensure_device())) return r;
  cudaStream_t st = as_stream(stream);
  return dtype == SB_F32 ? csr_dia_impl<float>(row_ptr, col, (const float*)val, N, nd, stride,
                                               offset, (float*)data, st)
                         : csr_dia_impl<double>(row_ptr, col, (const double*)val, N, nd, stride,
                                                offset, (double*)data, st);
}

int sb_coo_csc(int dtype, const int32_t* row, const int32_t* col, const void* val, int32_t N,
               int64_t nnz, int32_t* csc_col_ptr, int32_t* csc_row, void* csc_val,
               void* stream) {
  SB_TRACE("sb_coo_csc");
  // coo_csc is coo_csr with the roles of rows and columns swapped
  return sb_coo_csr(dtype, col, row, val, N, nnz, csc_col_ptr, csc_row, csc_val, stream);
}

}  // extern "C"
