// sb_buckets.cu -- the bucket sort behind coo_csr of unsorted input and the CSR
// transpose.
//
// A counting sort by single rows scatters 16-byte items over as many open
// places as there are rows: with 4M rows the places lie all over 700 MB, every
// store leaves half a sector in DRAM, and the scatter alone took 2.04 ms for
// 44M FP64 entries on B200 (1.4 GB at the copy rate: 0.22 ms).  Here a bucket is
// a range of 2^shift rows with 512 to 1024 entries on average, so the open
// places (one line a bucket, 62,500 of them) stay in L2 and leave it as whole
// lines; one block then sorts a bucket in shared memory and writes its piece of
// the CSR, row pointers included, coalesced.
//   count    bucket sizes (4 bytes an entry read)
//   scatter  items {key, value} into the buckets, in whatever order the cursors'
//            atomics give
//   sort     by the key: row in the bucket, column, input position.  The
//            position makes keys distinct and equal columns keep their input
//            order, so the result does not depend on the atomics' order.
// Measured on B200, coo_csr of shuffled entries without allocations: banded 4M
// x 11 FP64 2.95 -> 1.51 ms (scatter 0.82, sort 0.40, count 0.26), power-law 2M
// rows 3.4 -> 2.1; CSR transpose of 18M FP32 entries, 1M rows, 1.6 -> 0.67 (three
// 8-bit radix passes before).
#include <algorithm>

#include "sb_buckets.cuh"
#include "sb_prims.cuh"

namespace sb {
namespace {

constexpr int kThreads = 256;
constexpr int kItemsPerThread = 8;    // entries a thread counts
constexpr int kScatterItems = 4;      // and scatters
constexpr int kMaxShift = 8;          // rows of a bucket at most: 256
constexpr int kPad = 8;               // a counter has a 32-byte sector to itself
constexpr int kSmall = 1024;          // entries of a bucket that a small block sorts
constexpr int kMedium = 2048;         // a medium one
constexpr int kLarge = 8192;          // and a large one (128 KB of shared memory)
constexpr int kRankMax = 256;         // rows up to this long are sorted by ranks

struct __align__(16) Item {
  unsigned long long key;
  unsigned long long bits;  // the value's bits (FP32 in the low half)
};

__device__ __forceinline__ unsigned long long val_bits(float v) { return __float_as_uint(v); }
__device__ __forceinline__ unsigned long long val_bits(double v) {
  return (unsigned long long)__double_as_longlong(v);
}
__device__ __forceinline__ void bits_val(unsigned long long b, float& v) {
  v = __uint_as_float((unsigned)b);
}
__device__ __forceinline__ void bits_val(unsigned long long b, double& v) {
  v = __longlong_as_double((long long)b);
}

// Adds 1 to bucket b's (padded) counter for every lane that is `on` and returns the lane's place.
// Lanes of one bucket share an atomic where the input has neighbours together
// (rows in order, a banded matrix): 32 atomics on one address would queue up.
__device__ __forceinline__ int bucket_add(int* cnt, int b, bool on) {
  const int lane = threadIdx.x & 31;
  const int before = __shfl_up_sync(0xffffffffu, b, 1);
  const unsigned same = __ballot_sync(0xffffffffu, lane > 0 && b == before);
  if (__popc(same) < 8) return on ? atomicAdd(cnt + (size_t)b * kPad, 1) : 0;
  const unsigned peers = __match_any_sync(0xffffffffu, on ? b : -1);
  const int leader = __ffs(peers) - 1;
  int base = 0;
  if (on && lane == leader) base = atomicAdd(cnt + (size_t)b * kPad, __popc(peers));
  base = __shfl_sync(0xffffffffu, base, leader);
  return base + __popc(peers & ((1u << lane) - 1u));
}

// What the passes below leave for the host.
struct Flags {
  int bad;       // an index out of range
  int largest;   // bucket
  int listed[2]; // buckets for the medium and the large sort
  int unfit;     // the sample found a row beyond a bucket
  int slots;     // buckets beyond the large sort
  int runs[kMaxShift + 1];  // their largest run of 2^s rows
};

// One row beyond kLarge entries makes the buckets useless, and where it holds a
// good part of the entries, counting them costs more than all else, since its
// atomics queue up on one address.  A sample of kSamples entries, counted by
// rows in a hashed table, finds such a row before the count (a shuffled row of
// 4M among 18M entries: transpose 5.7 -> 1.6 ms on B200, the radix sort included;
// columns with a density of 1/c 6.9 -> 1.6, as rows of coo_csr 9.6 -> 2.5; 5 us for
// matrices without one).  `least` sightings stand for more than
// kLarge entries; a row that is missed, or met by chance, costs time only.
constexpr int kSamples = 16384;
constexpr long long kSampleFrom = 1 << 20;  // entries from which the sample pays

__global__ void __launch_bounds__(kThreads)
    bucket_sample(const int* __restrict__ row, long long nnz, int least, int* __restrict__ table,
                  Flags* __restrict__ flags) {
  const unsigned i = blockIdx.x * kThreads + threadIdx.x;
  const long long step = nnz / kSamples;
  const unsigned r = ld_stream(row + i * step + (i * 2654435761u >> 8) % (unsigned)step);
  if (atomicAdd(table + (r * 2654435761u) / (unsigned)(0x100000000ull / kSamples), 1) + 1 == least)
    flags->unfit = 1;
}

// Bucket sizes (cnt null, or a sample that found them useless: only the check);
// flags: an index out of range (with `check`; columns where they are given).
__global__ void __launch_bounds__(kThreads)
    bucket_count(const int* __restrict__ row, const int* __restrict__ col, long long nnz, int rows,
                 int cols, bool check, int shift, int* __restrict__ cnt,
                 Flags* __restrict__ flags) {
  const bool count = cnt && !flags->unfit;
  if (!count && !check) return;
  const long long base = (long long)blockIdx.x * kThreads * kItemsPerThread + threadIdx.x;
  int r[kItemsPerThread];
  bool bad = false;
#pragma unroll
  for (int u = 0; u < kItemsPerThread; ++u) {
    const long long k = base + u * kThreads;
    r[u] = k < nnz ? ld_stream(row + k) : 0;
    if (check && col && k < nnz) bad |= (unsigned)ld_stream(col + k) >= (unsigned)cols;
  }
#pragma unroll
  for (int u = 0; u < kItemsPerThread; ++u) {
    bool on = base + u * kThreads < nnz;
    if (check && (unsigned)r[u] >= (unsigned)rows) {
      bad = true;
      on = false;
      r[u] = 0;
    }
    if (count) bucket_add(cnt, r[u] >> shift, on);
  }
  if (bad) flags->bad = 1;
}

// The padded counts into start[0 .. n) (to be scanned; start[n] = 0); the
// largest into flags.
__global__ void bucket_sizes(const int* __restrict__ cnt, int n, int* __restrict__ start,
                             Flags* __restrict__ flags) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int c = i < n ? cnt[(size_t)i * kPad] : 0;
  if (i <= n) start[i] = c;
  const int m = __reduce_max_sync(0xffffffffu, c);
  if ((threadIdx.x & 31) == 0 && m > flags->largest) atomicMax(&flags->largest, m);
}
__global__ void bucket_cursors(const int* __restrict__ start, int n, int* __restrict__ cursor) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) cursor[(size_t)i * kPad] = start[i];
}

// Buckets beyond the large sort: their slots (slot[b], else -1), the entries of
// each of their rows, and from these the largest runs of 2^s rows, which tell
// how far the buckets have to be cut down, if that helps.
__global__ void bucket_slots(const int* __restrict__ cnt, int n, int* __restrict__ slot,
                             Flags* __restrict__ flags) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) slot[i] = cnt[(size_t)i * kPad] > kLarge ? atomicAdd(&flags->slots, 1) : -1;
}
__global__ void __launch_bounds__(kThreads)
    bucket_rows(const int* __restrict__ row, long long nnz, int shift,
                const int* __restrict__ slot, int* __restrict__ row_cnt) {
  const long long base = (long long)blockIdx.x * kThreads * kItemsPerThread + threadIdx.x;
#pragma unroll
  for (int u = 0; u < kItemsPerThread; ++u) {
    const long long k = base + u * kThreads;
    if (k >= nnz) continue;
    const int r = ld_stream(row + k), s = slot[r >> shift];
    if (s >= 0) atomicAdd(row_cnt + ((size_t)s << shift) + (r & ((1 << shift) - 1)), 1);
  }
}
__global__ void __launch_bounds__(1 << kMaxShift)
    bucket_runs(const int* __restrict__ row_cnt, int shift, Flags* __restrict__ flags) {
  __shared__ int sum[1 << kMaxShift];
  const int t = threadIdx.x;
  if ((int)blockIdx.x >= flags->slots) return;
  sum[t] = t < 1 << shift ? row_cnt[((size_t)blockIdx.x << shift) + t] : 0;
  for (int s = 0; s <= shift; ++s) {  // sum[i << s]: rows i << s to (i + 1) << s
    __syncthreads();
    const int v = t & ((1 << s) - 1) ? 0 : sum[t];
    if (v > kLarge) atomicMax(&flags->runs[s], v);
    __syncthreads();
    if (s < shift && (t & ((2 << s) - 1)) == 0) sum[t] = v + sum[t + (1 << s)];
  }
}

struct Bits {
  int shift;  // rows of a bucket, log2
  int col;    // bits of a column
  int pos;    // bits of an input position
};

template <typename T>
__device__ __forceinline__ Item make_item(int r, int c, long long k, T v, Bits b) {
  const unsigned local = (unsigned)r & ((1u << b.shift) - 1u);
  Item it;
  it.key = ((((unsigned long long)local << b.col) | (unsigned)c) << b.pos) |
           (unsigned long long)k;
  it.bits = val_bits(v);
  return it;
}
__device__ __forceinline__ void store_item(Item* p, Item it) {
  *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(it.key, it.bits);
}

template <typename T>
__global__ void __launch_bounds__(kThreads)
    bucket_scatter(const int* __restrict__ row, const int* __restrict__ col,
                   const T* __restrict__ val, long long nnz, Bits bits, int* __restrict__ cursor,
                   Item* __restrict__ items) {
  constexpr int U = kScatterItems;
  const long long base = (long long)blockIdx.x * kThreads * U + threadIdx.x;
  int r[U], c[U], p[U];
  T v[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const long long k = base + u * kThreads;
    const bool on = k < nnz;
    r[u] = on ? ld_stream(row + k) : 0;
    c[u] = on ? ld_stream(col + k) : 0;
    v[u] = on ? ld_stream(val + k) : T(0);
  }
#pragma unroll
  for (int u = 0; u < U; ++u)
    p[u] = bucket_add(cursor, r[u] >> bits.shift, base + u * kThreads < nnz);
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const long long k = base + u * kThreads;
    if (k < nnz) store_item(items + p[u], make_item(r[u], c[u], k, v[u], bits));
  }
}

// The same from a CSR, transposed: a warp walks the entries of `per` rows (at
// most 32), whose bounds its lanes hold; an entry's row by a search through them.
// Few rows of many entries take few rows to a warp, since every step waits for
// its atomics (transpose of 1000 rows of 65 entries, the whole call: 129 us with
// 32 rows to a warp, 85 with one; 30,000 rows 222 and 177).
template <typename T>
__global__ void __launch_bounds__(kThreads)
    bucket_scatter_csr(const int* __restrict__ csr_ptr, const int* __restrict__ col,
                       const T* __restrict__ val, int src_rows, int per, Bits bits,
                       int* __restrict__ cursor, Item* __restrict__ items) {
  const int lane = threadIdx.x & 31;
  const long long r0 = per * (((long long)blockIdx.x * kThreads + threadIdx.x) >> 5);
  if (r0 >= src_rows) return;
  const int n = (int)min((long long)per, src_rows - r0);
  // lane l: where row r0 + l ends (rows past the last: never)
  const int end = lane < n ? csr_ptr[r0 + lane + 1] : 0x7fffffff;
  const int first = csr_ptr[r0], last = __shfl_sync(0xffffffffu, end, n - 1);
  for (int k0 = first; k0 < last; k0 += 32) {
    const int k = k0 + lane;
    const bool on = k < last;
    const int c = on ? ld_stream(col + k) : 0;
    const T v = on ? ld_stream(val + k) : T(0);
    int r = 0;  // rows that end at or before k
#pragma unroll
    for (int step = 16; step > 0; step >>= 1)
      if (__shfl_sync(0xffffffffu, end, r + step - 1) <= k) r += step;
    const int p = bucket_add(cursor, c >> bits.shift, on);
    if (on) store_item(items + p, make_item(c, (int)(r0 + r), k, v, bits));
  }
}

// Sort of n keys with their bits by the whole block: the bitonic network whose
// comparators all put the smaller key first, so that the keys that would pad n
// to a power of two never move and their comparators are left out.
__device__ __forceinline__ void block_sort(unsigned long long* sk, unsigned long long* sv, int n) {
  auto exchange = [&](int i, int j) {
    if (j >= n) return;
    const unsigned long long ki = sk[i], kj = sk[j];
    if (ki > kj) {
      sk[i] = kj;
      sk[j] = ki;
      const unsigned long long t = sv[i];
      sv[i] = sv[j];
      sv[j] = t;
    }
  };
  int m = 2;
  while (m < n) m <<= 1;
  const int half = m >> 1;
  for (int size = 2; size <= m; size <<= 1) {
    // first against the mirror image in the block of `size`, then by strides
    for (int p = threadIdx.x; p < half; p += blockDim.x) {
      const int in = p & (size / 2 - 1), base = (p - in) * 2;
      exchange(base + in, base + size - 1 - in);
    }
    __syncthreads();
    for (int stride = size >> 2; stride > 0; stride >>= 1) {
      for (int p = threadIdx.x; p < half; p += blockDim.x) {
        const int i = ((p & ~(stride - 1)) << 1) | (p & (stride - 1));
        exchange(i, i + stride);
      }
      __syncthreads();
    }
  }
}

// One bucket per block: its rows counted, the items laid out row by row in
// shared memory, every item then ranked among its row's keys and stored at its
// place (rows of more than kRankMax entries are sorted by the block first).  The
// items are read twice, the second time from L1: holding them in registers
// instead halved the blocks per SM (44M entries: 0.62 against 0.38 ms).  CAP:
// entries that fit.  The small form takes all buckets and lists those beyond it
// for the medium one, which does the same for the large one (in_list null: all
// nbuckets; out_list null: nothing is larger).  Small blocks of 128 or 512
// threads or for up to 1536 or 2048 entries were slower.
template <typename T, int CAP, int TH>
__global__ void __launch_bounds__(TH, 2048 / TH)
    bucket_sort(const Item* __restrict__ items, const int* __restrict__ start, int nbuckets,
                int rows, Bits bits, const int* in_list, const int* n_in, int* out_list,
                int* n_out, int* __restrict__ out_ptr, int* __restrict__ out_col,
                T* __restrict__ out_val) {
  extern __shared__ __align__(16) unsigned long long sm[];
  unsigned long long* sk = sm;
  unsigned long long* sv = sm + CAP;
  __shared__ int cnt[(1 << kMaxShift) + 1];  // entries of a row, then where its next one goes
  __shared__ int longest;
  const int t = threadIdx.x;
  const int R = 1 << bits.shift;
  const int low = bits.col + bits.pos;
  const unsigned long long cmask = (1ull << bits.col) - 1ull;
  const int todo = in_list ? *n_in : nbuckets;
  for (int q = blockIdx.x; q < todo; q += gridDim.x) {
    const int b = in_list ? in_list[q] : q;
    const int s = start[b], n = start[b + 1] - s;
    if (n > CAP) {
      if (t == 0 && out_list) out_list[atomicAdd(n_out, 1)] = b;
      continue;
    }
    const int r0 = b << bits.shift;
    for (int r = t; r <= R; r += TH) cnt[r] = 0;
    __syncthreads();
    for (int k = t; k < n; k += TH) atomicAdd(cnt + (int)(__ldg(&items[s + k].key) >> low), 1);
    __syncthreads();
    // row starts, and with them the row pointers
    if (t < 32) {
      int carry = 0, top = 0;
      for (int r = t; r - t < R; r += 32) {
        const int v = r < R ? cnt[r] : 0;
        int x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, x, o);
          if (t >= o) x += y;
        }
        top = max(top, v);
        if (r < R) cnt[r] = carry + x - v;
        if (r < R && r0 + r < rows) out_ptr[r0 + r] = s + carry + x - v;
        carry += __shfl_sync(0xffffffffu, x, 31);
      }
      top = __reduce_max_sync(0xffffffffu, top);
      if (t == 0) longest = top;
      if (t == 0 && b == nbuckets - 1) out_ptr[rows] = s + n;
    }
    __syncthreads();
    for (int k = t; k < n; k += TH) {
      const ulonglong2 it = __ldg(reinterpret_cast<const ulonglong2*>(items + s + k));
      const int at = atomicAdd(cnt + (int)(it.x >> low), 1);
      sk[at] = it.x;
      sv[at] = it.y;
    }
    __syncthreads();
    // (cnt[r] is where row r ends by now)
    if (longest > kRankMax) {
      for (int r = 0; r < R; ++r) {
        const int lo = r ? cnt[r - 1] : 0, len = cnt[r] - lo;
        if (len > kRankMax) block_sort(sk + lo, sv + lo, len);
      }
    }
    // item k (in row order): the smaller keys of its row come before it.  The
    // lanes of a warp hold neighbouring items, so their places are a
    // permutation of nearly the same range and the stores stay coalesced.
    for (int k = t; k < n; k += TH) {
      const unsigned long long x = sk[k];
      const int r = (int)(x >> low);
      const int lo = r ? cnt[r - 1] : 0, hi = cnt[r];
      int at = k;
      if (hi - lo <= kRankMax) {
        at = lo;
#pragma unroll 4
        for (int j = lo; j < hi; ++j) at += sk[j] < x;
      }
      out_col[s + at] = (int)((x >> bits.pos) & cmask);
      T v;
      bits_val(sv[k], v);
      out_val[s + at] = v;
    }
    __syncthreads();
  }
}

unsigned blocks_for(long long n, int per) { return (unsigned)std::max(1LL, (n + per - 1) / per); }

}  // namespace

template <typename T>
int bucket_csr(const int* row, const int* col, const int* csr_ptr, const T* val, int rows,
               int cols, long long nnz, bool check, int* out_ptr, int* out_col, T* out_val,
               cudaStream_t st) {
  Bits bits;
  bits.col = prim::bits_for(cols > 0 ? cols - 1 : 0);
  bits.pos = prim::bits_for(nnz - 1);
  // 512 to 1024 entries a bucket, 256 rows at most; keys of at most 63 bits
  bits.shift = 0;
  while (bits.shift < kMaxShift && ((long long)nnz << (bits.shift + 1)) <= 1024LL * rows)
    ++bits.shift;
  bits.shift = std::min(bits.shift, 63 - bits.col - bits.pos);
  int *mem = nullptr, *cnt = nullptr, *start = nullptr, *list = nullptr;
  Item* items = nullptr;
  Flags* flags = nullptr;
  Flags hf = {};
  int nb = 0, r = SB_OK;
  const bool sample = nnz >= kSampleFrom;
  const size_t head = sizeof(Flags) + (sample ? sizeof(int) * kSamples : 0);  // and the table
  if ((r = scratch_alloc((void**)&flags, head, st))) return r;
  cudaError_t e = cudaMemsetAsync(flags, 0, head, st);
  if (e == cudaSuccess && sample) {
    const int least = std::max(24, (int)(1.25 * kLarge * kSamples / (double)nnz));
    bucket_sample<<<kSamples / kThreads, kThreads, 0, st>>>(row, nnz, least, (int*)(flags + 1),
                                                            flags);
    e = cudaGetLastError();
  }
  for (bool cut = false; e == cudaSuccess; cut = true) {
    nb = (int)((((long long)rows - 1) >> bits.shift) + 1);
    // cnt[nb] padded, start[nb + 1], lists[2][nb]; without memory for them the
    // entries are still checked
    const size_t ints = (size_t)nb * (kPad + 3) + 1;
    if (scratch_alloc((void**)&mem, sizeof(int) * ints, st)) mem = nullptr;
    cnt = mem;
    start = mem + (size_t)nb * kPad;
    list = start + nb + 1;
    if (mem) e = cudaMemsetAsync(mem, 0, sizeof(int) * (size_t)nb * kPad, st);
    if (e == cudaSuccess) {
      bucket_count<<<blocks_for(nnz, kThreads * kItemsPerThread), kThreads, 0, st>>>(
          row, col, nnz, rows, cols, check && !cut, bits.shift, cnt, flags);
      if (mem)
        bucket_sizes<<<blocks_for((long long)nb + 1, kThreads), kThreads, 0, st>>>(cnt, nb, start,
                                                                                flags);
      e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(&hf, flags, sizeof(hf), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) break;
    if (hf.bad) {
      set_error("index outside [0, %d)", rows);
      r = SB_EINVAL;
      break;
    }
    if (mem && !hf.unfit && hf.largest <= kLarge) break;
    r = kBucketsUnfit;
    if (!mem || hf.unfit || cut || bits.shift == 0) break;
    // buckets beyond shared memory (long rows next to one another, or one row):
    // fewer rows to a bucket, as few as it takes
    int* row_cnt = nullptr;
    const int most = (int)(nnz / kLarge) + 1;
    const size_t bytes = sizeof(int) * ((size_t)most << bits.shift);
    if (scratch_alloc((void**)&row_cnt, bytes, st)) break;
    e = cudaMemsetAsync(row_cnt, 0, bytes, st);
    if (e == cudaSuccess) {
      bucket_slots<<<blocks_for(nb, kThreads), kThreads, 0, st>>>(cnt, nb, list, flags);
      bucket_rows<<<blocks_for(nnz, kThreads * kItemsPerThread), kThreads, 0, st>>>(
          row, nnz, bits.shift, list, row_cnt);
      bucket_runs<<<most, 1 << kMaxShift, 0, st>>>(row_cnt, bits.shift, flags);
      e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(&hf, flags, sizeof(hf), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(flags, 0, sizeof(Flags), st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    scratch_free(row_cnt, st);
    if (e != cudaSuccess || hf.runs[0] > kLarge) break;
    while (bits.shift > 0 && hf.runs[bits.shift] > kLarge) --bits.shift;
    r = SB_OK;
    scratch_free(mem, st);
    mem = nullptr;
  }
  if (e != cudaSuccess) r = cuda_status(e, "bucket_csr (counts)");
  if (!r) r = prim::exclusive_scan(start, start, (long long)nb + 1, st);
  if (!r && scratch_alloc((void**)&items, sizeof(Item) * (size_t)nnz, st)) r = kBucketsUnfit;
  if (!r) {
    bucket_cursors<<<blocks_for(nb, kThreads), kThreads, 0, st>>>(start, nb, cnt);
    if (csr_ptr) {
      int per = 32;  // as many as leave 64 warps to an SM, 1 to 32
      while (per > 1 && (long long)per * 64 * sm_count() > cols) per >>= 1;
      bucket_scatter_csr<T><<<blocks_for(((long long)cols + per - 1) / per, kThreads / 32),
                              kThreads, 0, st>>>(csr_ptr, row, val, cols, per, bits, cnt, items);
    } else {
      bucket_scatter<T><<<blocks_for(nnz, kThreads * kScatterItems), kThreads, 0, st>>>(
          row, col, val, nnz, bits, cnt, items);
    }
    e = cudaGetLastError();
    auto small = bucket_sort<T, kSmall, kThreads>;
    auto medium = bucket_sort<T, kMedium, 512>;
    auto large = bucket_sort<T, kLarge, 1024>;
    if (e == cudaSuccess) {
      small<<<std::min(nb, 1 << 20), kThreads, 16 * kSmall, st>>>(
          items, start, nb, rows, bits, nullptr, nullptr, list, flags->listed, out_ptr, out_col,
          out_val);
      e = cudaGetLastError();
    }
    if (e == cudaSuccess && hf.largest > kSmall) {
      medium<<<4 * sm_count(), 512, 16 * kMedium, st>>>(
          items, start, nb, rows, bits, list, flags->listed, list + nb, flags->listed + 1, out_ptr,
          out_col, out_val);
      e = cudaGetLastError();
    }
    if (e == cudaSuccess && hf.largest > kMedium) {
      e = cudaFuncSetAttribute((const void*)large, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               16 * kLarge);
      if (e == cudaSuccess) {
        large<<<sm_count(), 1024, 16 * kLarge, st>>>(items, start, nb, rows, bits, list + nb,
                                                     flags->listed + 1, nullptr, nullptr, out_ptr,
                                                     out_col, out_val);
        e = cudaGetLastError();
      }
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) r = cuda_status(e, "bucket_csr");
  }
  if (items) scratch_free(items, st);
  if (mem) scratch_free(mem, st);
  scratch_free(flags, st);
  return r;
}

template int bucket_csr<float>(const int*, const int*, const int*, const float*, int, int,
                               long long, bool, int*, int*, float*, cudaStream_t);
template int bucket_csr<double>(const int*, const int*, const int*, const double*, int, int,
                                long long, bool, int*, int*, double*, cudaStream_t);

}  // namespace sb
