// column_mask.cuh -- which columns hold no nonzero stored value (the dangling
// vertices of a PageRank matrix).
//
// Marking a byte per stored entry queues up at a power-law graph's hot columns
// (R-MAT 2^17, 2 million entries: 89 us; reading the byte first to spare the
// store: 320 us on 2^16, the reads wait behind the stores).  The columns
// with a stored entry depend on the pattern alone, so they are marked once per
// handle; a solve then only looks for stored zeros (a streaming read of the
// values, 5 us) and marks again when there are any.
#pragma once

#include <algorithm>

#include "common.cuh"

namespace tbsla {

inline int mask_grid(int64_t n) { return (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 152 * 8)); }

// mask[c - f_col] = 0 for every entry with a nonzero value (vals NULL: every
// entry); when: unless NULL, only if *when is nonzero
template <typename V>
__global__ void __launch_bounds__(256) column_mark_kernel(const int *__restrict__ cols, const V *__restrict__ vals,
                                                         int64_t n, int f_col, int n_col, const int *when,
                                                         unsigned char *mask) {
  if (when && !*when) return;
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
    const int c = cols[k] - f_col;
    if ((!vals || vals[k] != V(0)) && c >= 0 && c < n_col) mask[c] = 0;
  }
}

// *zeros = 1 when a value is 0
template <typename V>
__global__ void __launch_bounds__(256) zero_value_kernel(const V *__restrict__ vals, int64_t n, int *zeros) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  bool any = false;
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += 4 * stride) {
    #pragma unroll
    for (int u = 0; u < 4; ++u) any |= k + u * stride < n && vals[k + u * stride] == V(0);
  }
  if (__any_sync(0xffffffffu, any) && (threadIdx.x & 31) == 0) *zeros = 1;
}

// mask = every column without entries (when no value is 0), else all ones
__global__ void __launch_bounds__(256) mask_start_kernel(const unsigned char *__restrict__ pattern, int n_col,
                                                         const int *zeros, unsigned char *mask);

// A's columns without a stored entry (1) or with one (0), built on first use
tbsla_status_t column_pattern(tbsla_matrix *A, const unsigned char **pattern);

// mask[c] = 1 for the columns of CSR / COO handle A without a nonzero value in
// `vals`, 0 for the others; zeros: one int of scratch
template <typename V>
tbsla_status_t column_mask(tbsla_matrix *A, const V *vals, unsigned char *mask, int *zeros, cudaStream_t s) {
  const unsigned char *pattern = nullptr;
  TB_TRY(column_pattern(A, &pattern));
  const int64_t n = A->stored;
  TB_CUDA(cudaMemsetAsync(zeros, 0, sizeof(int), s));
  if (n) zero_value_kernel<V><<<(int)std::max<int64_t>(1, std::min<int64_t>((n + 1023) / 1024, 152 * 8)), 256, 0, s>>>(vals, n, zeros);
  mask_start_kernel<<<mask_grid(A->n_col), 256, 0, s>>>(pattern, A->n_col, zeros, mask);
  if (n) column_mark_kernel<V><<<mask_grid(n), 256, 0, s>>>(A->idx1, vals, n, A->f_col, A->n_col, zeros, mask);
  TB_CUDA(cudaGetLastError());
  return TBSLA_OK;
}

}  // namespace tbsla
