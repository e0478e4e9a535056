// sb_buckets.cuh -- entries in any order into a CSR with every row ordered by
// (column, input position): the stable counting sort of coo_csr and of the
// CSR transpose.
#pragma once

#include "sb_common.cuh"

namespace sb {

// Returned by the bucket sort, with nothing written but the indices checked,
// when the entries do not suit it (a row beyond shared memory) or its scratch
// memory cannot be had: the caller's radix sort takes over.
constexpr int kBucketsUnfit = 1;

// Entry k is (row[k], col[k], val[k]); with csr_ptr (and row) given instead of
// col, entry k of a CSR is taken as (row[k] = its column, its row, val[k]),
// which is the transpose.  rows, cols: the index ranges of the result.  The
// indices are checked where `check` is set (SB_EINVAL).  Returns after the work.
template <typename T>
int bucket_csr(const int* row, const int* col, const int* csr_ptr, const T* val, int rows,
               int cols, long long nnz, bool check, int* out_ptr, int* out_col, T* out_val,
               cudaStream_t st);

}  // namespace sb
