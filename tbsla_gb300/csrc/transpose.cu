// transpose.cu -- the CSR differentiation helpers: the transposed copy
// (A^T x), the gradient of y = A x with respect to the values (the outer
// product a b^T sampled on the sparsity pattern), and value replacement.
//
// The transposed copy is an ordinary CSR handle (so A^T x runs the same
// kernels as A x).  It is built once, on the device: entries sorted by column,
// stably, so that row j of the copy lists column j's entries in increasing
// row order.  transpose_perm maps its entries back to A's, so new values of A
// reach the copy by a gather on the device.
#include <vector>

#include "device_sort.cuh"
#include "product.cuh"

namespace tbsla {

tbsla_status_t spmv_dispatch(const tbsla_matrix *A, tbsla_dtype_t store, tbsla_dtype_t xt, const void *x,
                             tbsla_dtype_t yt, void *y, int vect_incr, cudaStream_t s);
tbsla_status_t sell_refresh(tbsla_matrix *A, cudaStream_t s);

namespace {

// out[k] = scale * a[row(k)] * b[col(k) - f_col].  A warp takes segments of
// kGradSeg consecutive entries whatever their rows, so the column loads and
// gradient stores are coalesced and hub rows spread over warps; seg_row[s] is
// the row of segment s's first entry.  The lanes hold the ends of the 32 rows
// from there on, and a lane finds its entry's row by a binary search over them
// (shuffles); a segment that leaves those 32 rows goes on with the next 32, as
// long as they end at least kGradWindow of its entries.  Where rows with entries lie
// further apart, the lanes search the row pointer up to the next segment's row
// for each of their entries, the four searches in flight together: one warp
// walked a run of 4 million empty rows inside its segment 32 at a time, 54 ms
// for a gradient of 10 thousand entries.
// The segment's index loads, then its gathers (b with the handle's L2 policy
// for x, TBSLA_TUNE_X_L2_KEEP), are in flight together.  One row per thread
// for short rows and 4 to 32 lanes per long row left R-MAT 2^16 at 175 us, 120
// of them its hub rows.
constexpr int kGradSeg = 128, kGradWindow = 16;

template <typename T>
__global__ void __launch_bounds__(256) grad_segment_kernel(int rows, int64_t nnz, const int *__restrict__ seg_row,
                                                          const int *__restrict__ rowptr,
                                                          const int *__restrict__ colidx, int f_col,
                                                          const T *__restrict__ a, const T *__restrict__ b,
                                                          T scale, T *__restrict__ out, XKeep b_keep) {
  constexpr int U = kGradSeg / 32;
  const int lane = threadIdx.x & 31;
  const uint64_t keep = policy_keep(b_keep, b);
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w * kGradSeg < nnz; w += nwarps) {
    const int64_t e0 = w * kGradSeg;
    const int n = (int)min((int64_t)kGradSeg, nnz - e0);
    int r0 = __ldg(seg_row + w);
    int col[U];
    T bv[U];
    #pragma unroll
    for (int u = 0; u < U; ++u) col[u] = 32 * u + lane < n ? ld_stream(colidx + e0 + 32 * u + lane) : f_col;
    #pragma unroll
    for (int u = 0; u < U; ++u) bv[u] = 32 * u + lane < n ? ld_keep(b + (col[u] - f_col), keep) : T(0);
    int done = 0;  // entries of the segment in rows before r0
    for (bool dense = true; dense && done < n;) {
      const int r = min(r0 + lane, rows - 1);
      // the end of row r0 + lane, relative to the segment
      const int end = (int)min((int64_t)__ldg(rowptr + r + 1) - e0, (int64_t)kGradSeg);
      const T ar = scale * __ldg(a + r);
      const int last = min(__shfl_sync(0xffffffffu, end, 31), n);
      #pragma unroll
      for (int u = 0; u < U; ++u) {
        const int e = 32 * u + lane;
        if (32 * u >= last || 32 * u + 32 <= done) continue;  // uniform: no entry of these rows here
        int j = 0;  // rows that end at or before e
        #pragma unroll
        for (int step = 16; step >= 1; step >>= 1) {
          const int v = __shfl_sync(0xffffffffu, end, j + step - 1);
          if (v <= e) j += step;
        }
        const T arow = __shfl_sync(0xffffffffu, ar, j);
        if (e >= done && e < last) __stcs(out + e0 + e, arow * bv[u]);
      }
      dense = last - done >= kGradWindow;
      done = last;
      r0 += 32;
    }
    if (done < n) {
      // the last row from r0 on that begins at or before the entry; entry `done` is in
      // one of them, so r0 is a row and begins there or before
      int row[U];
      #pragma unroll
      for (int u = 0; u < U; ++u) row[u] = r0;
      for (int len = e0 + n < nnz ? __ldg(seg_row + w + 1) - r0 + 1 : rows - r0; len > 1; len -= len >> 1) {
        #pragma unroll
        for (int u = 0; u < U; ++u)
          if (__ldg(rowptr + row[u] + (len >> 1)) <= e0 + 32 * u + lane) row[u] += len >> 1;
      }
      #pragma unroll
      for (int u = 0; u < U; ++u) {
        const int e = 32 * u + lane;
        if (e >= done && e < n) __stcs(out + e0 + e, scale * __ldg(a + row[u]) * bv[u]);
      }
    }
  }
}

// All rows short and in order: a warp takes 32 rows and strides its lanes over
// their entries, four strides at a time, so the rows' ends are loaded once for
// all of them and their index is found without seg_row.  On even rows the
// segments above pay for the ends of 32 rows at every 128 entries: 16 entries a
// row, FP32, 2^20 / 2^22 / 2^24 rows: 37 / 121 / 460 us here, 51 / 200 / 786
// there (four segments a warp: 45 / 152 / 571); 2^16 rows 13 and 11.
template <typename T>
__global__ void __launch_bounds__(256) grad_tile_kernel(int rows, const int *__restrict__ rowptr,
                                                          const int *__restrict__ colidx, int f_col,
                                                          const T *__restrict__ a, const T *__restrict__ b,
                                                          T scale, T *__restrict__ out, XKeep b_keep) {
  constexpr int U = 4;
  const int lane = threadIdx.x & 31;
  const uint64_t keep = policy_keep(b_keep, b);
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w * 32 < rows; w += nwarps) {
    const int r0 = (int)(w * 32);
    const int mine = min(r0 + lane, rows);
    const int start = __ldg(rowptr + mine);                    // row start of row r0 + lane
    const T ar = r0 + lane < rows ? scale * a[r0 + lane] : T(0);
    const int first = __shfl_sync(0xffffffffu, start, 0);
    const int end = __ldg(rowptr + min(r0 + 32, rows));
    for (int e0 = first; e0 < end; e0 += 32 * U) {
      int col[U];
      T bv[U];
      #pragma unroll
      for (int u = 0; u < U; ++u) {
        const int e = e0 + 32 * u + lane;
        col[u] = e < end ? ld_stream(colidx + e) : f_col;
      }
      #pragma unroll
      for (int u = 0; u < U; ++u) {
        const int e = e0 + 32 * u + lane;
        bv[u] = e < end ? ld_keep(b + (col[u] - f_col), keep) : T(0);
      }
      #pragma unroll
      for (int u = 0; u < U; ++u) {
        const int e = e0 + 32 * u + lane;
        int j = 0;  // largest lane index with start <= e
        #pragma unroll
        for (int step = 16; step >= 1; step >>= 1) {
          const int cand = j + step;
          const int v = __shfl_sync(0xffffffffu, start, cand & 31);
          if (cand < 32 && v <= e) j = cand;
        }
        const T arow = __shfl_sync(0xffffffffu, ar, j);
        if (e < end) __stcs(out + e, arow * bv[u]);
      }
    }
  }
}

// seg_row[s] = the row of entry s * kGradSeg
__global__ void grad_segments_kernel(int rows, const int *__restrict__ rowptr, int *__restrict__ seg_row) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += (int64_t)gridDim.x * blockDim.x) {
    const int a = rowptr[r], b = rowptr[r + 1];
    for (int64_t s = ((int64_t)a + kGradSeg - 1) / kGradSeg; s * kGradSeg < b; ++s) seg_row[s] = (int)r;
  }
}

// entry k' of the transposed copy's stores from new values at perm[k'], four
// gathers of a thread in flight
template <typename S>
__global__ void __launch_bounds__(256) permute_values_kernel(const S *__restrict__ src, const int *__restrict__ perm,
                                                            int64_t n, double *__restrict__ f64,
                                                            float *__restrict__ f32,
                                                            __nv_bfloat16 *__restrict__ bf16) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += 4 * stride) {
    S v[4];
    #pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = k + u * stride < n ? __ldg(src + ld_stream(perm + k + u * stride)) : S(0);
    #pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int64_t at = k + u * stride;
      if (at >= n) break;
      if (f64) f64[at] = (double)v[u];
      if (f32) f32[at] = sizeof(S) == 8 ? __double2float_rn((double)v[u]) : (float)v[u];
      if (bf16) bf16[at] = __double2bfloat16((double)v[u]);
    }
  }
}

// key = column of the block, entry = position
__global__ void __launch_bounds__(256) column_keys_kernel(const int *__restrict__ col, int f_col, int64_t n,
                                                         uint32_t *__restrict__ keys, int *__restrict__ entries) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
    keys[k] = (uint32_t)(col[k] - f_col);
    entries[k] = (int)k;
  }
}

bool csr_direct(const tbsla_matrix *A) { return A && A->format == TBSLA_FMT_CSR && A->csr_variant == 0; }

template <typename T>
tbsla_status_t grad_values(const tbsla_matrix *A, const T *a, const T *b, T scale, T *out, cudaStream_t s) {
  if (A->stored == 0 || A->rows == 0) return TBSLA_OK;
  if (A->short_rows == nullptr && A->n_short == A->rows) {  // every row short, in order
    grad_tile_kernel<T><<<(int)std::min<int64_t>(((int64_t)A->rows + 255) / 256, 152 * 64), 256, 0, s>>>(
        A->rows, A->idx0, A->idx1, A->f_col, a, b, scale, out, xkeep_of<T>(A));
    TB_CUDA(cudaGetLastError());
    return TBSLA_OK;
  }
  const int64_t segs = (A->stored + kGradSeg - 1) / kGradSeg;
  grad_segment_kernel<T><<<(int)std::min<int64_t>((segs + 7) / 8, 152 * 64), 256, 0, s>>>(
      A->rows, A->stored, A->seg_row, A->idx0, A->idx1, A->f_col, a, b, scale, out, xkeep_of<T>(A));
  TB_CUDA(cudaGetLastError());
  return TBSLA_OK;
}

}  // namespace

// The segments' rows of a CSR handle, at its creation (the row structure only)
tbsla_status_t grad_segments(tbsla_matrix *A) {
  if (A->stored == 0 || A->rows == 0) return TBSLA_OK;
  const int64_t segs = (A->stored + kGradSeg - 1) / kGradSeg;
  TB_TRY(dev_alloc(A, (void **)&A->seg_row, (size_t)segs * sizeof(int)));
  grad_segments_kernel<<<(int)std::min<int64_t>(((int64_t)A->rows + 255) / 256, 152 * 16), 256>>>(A->rows, A->idx0,
                                                                                               A->seg_row);
  TB_CUDA(cudaGetLastError());
  return TBSLA_OK;
}

// The transposed copy of a CSR handle, built on first use.
tbsla_status_t ensure_transpose(tbsla_matrix *A, tbsla_matrix **T) {
  std::lock_guard<std::mutex> lk(A->first_use);
  if (A->transpose) {
    *T = A->transpose;
    return TBSLA_OK;
  }
  TB_CHECK(A->format == TBSLA_FMT_CSR, "the transpose needs a CSR handle");
  TB_CHECK(A->values[0], "the transpose needs the F64 value store");
  TB_CUDA(cudaSetDevice(A->device));
  const int ncol = A->n_col;
  const int64_t nnz = A->stored;
  const int grid = entry_grid(nnz);
  tbsla_matrix *B = new_matrix(TBSLA_FMT_CSR);
  if (!B) return fail(TBSLA_ERR_OOM, "host allocation failed");
  struct Guard {
    tbsla_matrix *B;
    int *perm = nullptr;
    ~Guard() {
      if (perm) cudaFree(perm);
      if (B) free_matrix(B);
    }
  } guard{B};
  B->device = A->device;
  TB_CUDA(cudaSetDevice(A->device));
  B->n_row = ncol;
  B->n_col = A->n_row;
  B->rows = ncol;
  B->stored = nnz;
  TB_TRY(alloc_ints(B, &B->idx0, (int64_t)ncol + 1));
  TB_CUDA(cudaDeviceSynchronize());  // A's values and arrays are in place, whichever stream wrote them
  {
    SortScratch sc;
    SortPairs<uint32_t> p;
    TB_TRY(p.get(sc, nnz));
    if (nnz) {
      column_keys_kernel<<<grid, 256>>>(A->idx1, A->f_col, nnz, p.keys, p.entries);
      TB_TRY(p.sort(sc, key_bits((uint64_t)std::max(ncol - 1, 0))));
    }
    key_starts_kernel<<<entry_grid((int64_t)ncol + 1), 256>>>(p.keys, nnz, (int64_t)ncol, B->idx0);
    TB_CUDA(cudaGetLastError());
    sc.give(p.entries);
    guard.perm = p.entries;
  }
  TB_TRY(alloc_ints(B, &B->idx1, nnz));
  if (nnz) {
    SortScratch sc;
    int *row = nullptr;
    TB_TRY(sc.get(&row, nnz));
    entry_rows_kernel<<<152 * 16, 256>>>(A->rows, A->idx0, row);
    take_kernel<<<grid, 256>>>(row, guard.perm, nnz, B->idx1);
    int last = 0;  // the entries come in row order: the last one's row is the largest
    TB_CUDA(cudaMemcpy(&last, row + nnz - 1, sizeof last, cudaMemcpyDeviceToHost));
    B->x_extent = (int64_t)last + 1;
  }
  TB_TRY(take_values(B, A, guard.perm));
  std::vector<int> tp((size_t)ncol + 1);
  TB_CUDA(cudaMemcpy(tp.data(), B->idx0, tp.size() * sizeof(int), cudaMemcpyDeviceToHost));
  TB_TRY(csr_bins(B, tp));
  B->x_keep = A->x_keep;
  B->x_keep_range = A->x_keep_range;
  B->short_mode = A->short_mode;
  B->pr_polls = A->pr_polls;
  int *d_perm = guard.perm;
  guard.perm = nullptr;
  guard.B = nullptr;
  A->transpose = B;
  A->transpose_perm = d_perm;
  *T = B;
  return TBSLA_OK;
}

// After A's values changed to d_values: the copy's stores follow in one pass
// (and, where it has one, its ELL-layout copy)
tbsla_status_t transpose_refresh(tbsla_matrix *A, tbsla_dtype_t type, const void *d_values, cudaStream_t s) {
  if (!A->transpose || !A->stored) return TBSLA_OK;
  tbsla_matrix *T = A->transpose;
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((A->stored + 1023) / 1024, 152 * 32));
  double *f64 = static_cast<double *>(T->values[0]);
  float *f32 = static_cast<float *>(T->values[1]);
  __nv_bfloat16 *bf16 = static_cast<__nv_bfloat16 *>(T->values[2]);
  if (type == TBSLA_F64)
    permute_values_kernel<double><<<grid, 256, 0, s>>>(static_cast<const double *>(d_values), A->transpose_perm,
                                                       A->stored, f64, f32, bf16);
  else
    permute_values_kernel<float><<<grid, 256, 0, s>>>(static_cast<const float *>(d_values), A->transpose_perm,
                                                      A->stored, f64, f32, bf16);
  TB_CUDA(cudaGetLastError());
  return sell_refresh(T, s);
}

tbsla_status_t grad_values_f64(const tbsla_matrix *A, const double *a, const double *b, double scale, double *out,
                               cudaStream_t s) {
  return grad_values<double>(A, a, b, scale, out, s);
}

}  // namespace tbsla

using namespace tbsla;

extern "C" {

tbsla_status_t tbsla_spmv_transpose_ex(const tbsla_matrix_t *A, tbsla_dtype_t store, tbsla_dtype_t x_type,
                                       const void *d_x, tbsla_dtype_t y_type, void *d_y, void *stream) {
  TB_CHECK(A, "matrix is NULL");
  TB_CHECK(A->format == TBSLA_FMT_CSR, "tbsla_spmv_transpose_ex needs a CSR handle");
  tbsla_matrix *T = nullptr;
  TB_TRY(ensure_transpose(const_cast<tbsla_matrix *>(A), &T));
  return spmv_dispatch(T, store, x_type, d_x, y_type, d_y, 0, (cudaStream_t)stream);
}

tbsla_status_t tbsla_csr_grad_values(const tbsla_matrix_t *A, tbsla_dtype_t type, const void *d_a, const void *d_b,
                                     double scale, void *d_out, void *stream) {
  TB_CHECK(A, "matrix is NULL");
  TB_CHECK(csr_direct(A), "tbsla_csr_grad_values needs a CSR handle (default kernel variant)");
  TB_CHECK(A->stored == 0 || (d_a && d_b && d_out), "NULL vector");
  TB_CUDA(cudaSetDevice(A->device));
  if (type == TBSLA_F64)
    return grad_values<double>(A, static_cast<const double *>(d_a), static_cast<const double *>(d_b), scale,
                               static_cast<double *>(d_out), (cudaStream_t)stream);
  TB_CHECK(type == TBSLA_F32, "type must be TBSLA_F64 or TBSLA_F32");
  return grad_values<float>(A, static_cast<const float *>(d_a), static_cast<const float *>(d_b), (float)scale,
                            static_cast<float *>(d_out), (cudaStream_t)stream);
}

}  // extern "C"

// ------------------------------------------------------- normalize_columns
// MatrixCSR::normalize_columns (src/cpp/matrix/MatrixCSR.cpp:423-435) on the
// device: column sums accumulated from 0 in the order of the reference's
// loop (rows ascending, then stored order) -- the transposed copy lists each
// column's entries in exactly that order, so one thread per column repeats
// the reference's additions -- then every value divided by its column's sum
// (IEEE division, as the host's).  The values then go through
// tbsla_matrix_set_values, which refreshes every derived copy.
namespace tbsla {
namespace {

__global__ void colsum_kernel(const int *__restrict__ tp, const double *__restrict__ tv, int ncol,
                              double *__restrict__ sum) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < ncol; j += gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int k = tp[j]; k < tp[j + 1]; ++k) s += tv[k];
    sum[j] = s;
  }
}

__global__ void divide_kernel(const double *__restrict__ v, const int *__restrict__ ci, int f_col, int64_t n,
                              const double *__restrict__ sum, double *__restrict__ out) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x)
    out[k] = v[k] / sum[ci[k] - f_col];
}

}  // namespace
}  // namespace tbsla

extern "C" tbsla_status_t tbsla_csr_normalize_columns(tbsla_matrix_t *A, void *stream) {
  TB_CHECK(A, "matrix is NULL");
  TB_CHECK(A->format == TBSLA_FMT_CSR, "tbsla_csr_normalize_columns needs a CSR handle");
  TB_CHECK(A->values[0], "the F64 value store is needed");
  TB_CUDA(cudaSetDevice(A->device));
  if (A->stored == 0) return TBSLA_OK;
  tbsla_matrix *T = nullptr;
  TB_TRY(ensure_transpose(A, &T));
  cudaStream_t s = (cudaStream_t)stream;
  double *sum = nullptr, *out = nullptr;
  const int ncol = std::max(A->n_col, 1);
  if (cudaMalloc(&sum, (size_t)ncol * 8) != cudaSuccess || cudaMalloc(&out, (size_t)A->stored * 8) != cudaSuccess) {
    cudaGetLastError();
    if (sum) cudaFree(sum);
    return fail(TBSLA_ERR_OOM, "normalize_columns scratch");
  }
  tbsla_status_t st = TBSLA_OK;
  colsum_kernel<<<std::max(1, std::min((T->rows + 255) / 256, 152 * 16)), 256, 0, s>>>(
      T->idx0, static_cast<const double *>(T->values[0]), T->rows, sum);
  divide_kernel<<<152 * 8, 256, 0, s>>>(static_cast<const double *>(A->values[0]), A->idx1, A->f_col, A->stored, sum,
                                       out);
  if (cudaGetLastError() != cudaSuccess) st = fail(TBSLA_ERR_CUDA, "normalize_columns kernels failed");
  if (st == TBSLA_OK) st = tbsla_matrix_set_values(A, TBSLA_F64, out, stream);
  cudaStreamSynchronize(s);
  cudaFree(sum);
  cudaFree(out);
  return st;
}
