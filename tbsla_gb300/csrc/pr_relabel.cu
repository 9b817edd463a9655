// pr_relabel.cu -- PageRank on a relabelled copy of the graph.
//
// A PageRank sweep gathers the iterate at the column of every stored entry.
// On power-law graphs (R-MAT) most gathers land on a small set of hot
// vertices, but in the generator's labels these are spread over the whole
// index range: every hot value shares its 32-byte sector with cold ones, so
// the hot set needs several times its size in L2 and most gathers go to
// DRAM.  Relabelling the vertices in decreasing out-degree (stored entries
// per column) packs the hot values together.  The relabelling is symmetric
// (rows and columns), so a sweep on the copy is the sweep on the original
// with permuted vectors; teleport, dangling mass, residual and maximum are
// permutation invariant, and the result is gathered back to the original
// labels.  Each row's entries are sorted by their new column, so the lanes
// of a long row's group gather neighbouring values of the hot set in one
// load instruction (R-MAT 2^24: 1.54 -> 1.40 ms per FP64 sweep against the
// rows in their original order); sums differ from the original labels'
// only by rounding.
//
// Order: out-degree class (floor(log2(out-degree + 1)), descending) first,
// which keeps the hot values together; inside a class, in-degree (the row
// length) descending, so that neighbouring rows have similar lengths and
// the thread-per-row kernel's warps run similar trip counts.
//
// The copy is built once per handle on the device (a stable sort of the
// vertices by degree, then of the entries by new row and column), an ordinary
// CSR handle with the same value stores.
#include <algorithm>
#include <vector>

#include "common.cuh"
#include "device_sort.cuh"

namespace tbsla {

namespace {

constexpr int kBandSamples = 4096;
constexpr int kBandWidth = 1024;

// entries within kBandWidth of the diagonal, and all entries, on
// kBandSamples rows spread evenly (one warp per sampled row)
__global__ void band_sample_kernel(const int *__restrict__ rowptr, const int *__restrict__ colidx, int n,
                                   int f_col, unsigned long long *cnt) {
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (w >= kBandSamples) return;
  const int r = (int)(((long long)w * n) / kBandSamples);
  const int a = rowptr[r], b = rowptr[r + 1];
  unsigned long long near = 0, all = 0;
  for (int k = a + lane; k < b; k += 32) {
    ++all;
    if (abs(colidx[k] - f_col - r) <= kBandWidth) ++near;
  }
  for (int o = 16; o > 0; o >>= 1) {
    near += __shfl_down_sync(0xffffffffu, near, o);
    all += __shfl_down_sync(0xffffffffu, all, o);
  }
  if (lane == 0) {
    atomicAdd(cnt, near);
    atomicAdd(cnt + 1, all);
  }
}

// deg[c - f_col] += 1 for every stored entry
__global__ void column_count_kernel(const int *__restrict__ colidx, int64_t nnz, int f_col, int *deg) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < nnz; k += (int64_t)gridDim.x * blockDim.x)
    atomicAdd(deg + (colidx[k] - f_col), 1);  // columns are in [f_col, f_col + n) (candidate())
}

// key: out-degree class descending, then in-degree (row length) descending;
// class = floor(log2(out-degree + 1))
__global__ void vertex_keys_kernel(const int *__restrict__ deg, const int *__restrict__ rowptr, int n, int top_cls,
                                   uint64_t *__restrict__ keys, int *__restrict__ verts) {
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
    const int cls = 31 - __clz(deg[v] + 1);
    keys[v] = (uint64_t)(top_cls - cls) << 32 | (uint32_t)(0x7fffffff - (rowptr[v + 1] - rowptr[v]));
    verts[v] = (int)v;
  }
}

// newid[order[i]] = i
__global__ void new_labels_kernel(const int *__restrict__ order, int n, int *__restrict__ newid) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    newid[order[i]] = (int)i;
}

// key = new column of the entry, entry = position
__global__ void new_column_keys_kernel(const int *__restrict__ col, int f_col, const int *__restrict__ newid,
                                       int64_t nnz, uint32_t *__restrict__ keys, int *__restrict__ entries) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < nnz; k += (int64_t)gridDim.x * blockDim.x) {
    keys[k] = (uint32_t)newid[col[k] - f_col];
    entries[k] = (int)k;
  }
}

// rows[k] = newid[rows[k]]
__global__ void new_rows_kernel(const int *__restrict__ newid, int64_t nnz, uint32_t *__restrict__ rows) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < nnz; k += (int64_t)gridDim.x * blockDim.x)
    rows[k] = (uint32_t)newid[rows[k]];
}

// out[k] = the new column of entry order[k]
__global__ void take_columns_kernel(const int *__restrict__ col, int f_col, const int *__restrict__ newid,
                                    const int *__restrict__ order, int64_t nnz, int *__restrict__ out) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < nnz; k += (int64_t)gridDim.x * blockDim.x)
    out[k] = newid[col[order[k]] - f_col];
}

int cls_max(int maxdeg) { return 31 - __builtin_clz((unsigned)maxdeg + 1u); }

bool candidate(const tbsla_matrix *A) {
  return A->format == TBSLA_FMT_CSR && A->csr_variant == 0 && A->n_row == A->n_col && A->rows == A->n_row &&
         A->stored > 0 && A->values[0] != nullptr && A->x_extent <= A->n_col;
}

// banded matrices (cqmat, cdiag) already gather locally
tbsla_status_t banded(const tbsla_matrix *A, bool *is_banded) {
  unsigned long long *d = nullptr, h[2] = {0, 0};
  TB_CUDA(cudaMalloc(&d, 2 * sizeof(unsigned long long)));
  cudaMemset(d, 0, 2 * sizeof(unsigned long long));
  band_sample_kernel<<<kBandSamples * 32 / 256, 256>>>(A->idx0, A->idx1, A->n_row, A->f_col, d);
  const cudaError_t e = cudaMemcpy(h, d, sizeof h, cudaMemcpyDeviceToHost);
  cudaFree(d);
  TB_CUDA(e);
  *is_banded = h[1] == 0 || 2 * h[0] >= h[1];
  return TBSLA_OK;
}

tbsla_status_t build(tbsla_matrix *A, bool check_skew, bool *built) {
  *built = false;
  const int n = A->n_row;
  const int64_t nnz = A->stored;
  // out-degrees
  SortScratch degrees;
  int *d_deg = nullptr;
  TB_TRY(degrees.get(&d_deg, n));
  TB_CUDA(cudaDeviceSynchronize());  // A's values and arrays are in place, whichever stream wrote them
  TB_CUDA(cudaMemset(d_deg, 0, (size_t)n * sizeof(int)));
  column_count_kernel<<<152 * 8, 256>>>(A->idx1, nnz, A->f_col, d_deg);
  std::vector<int> deg((size_t)n);
  TB_CUDA(cudaMemcpy(deg.data(), d_deg, (size_t)n * sizeof(int), cudaMemcpyDeviceToHost));
  const int maxdeg = *std::max_element(deg.begin(), deg.end());
  if (check_skew) {
    // entries in the columns of the n/10 vertices of highest out-degree
    std::vector<int64_t> hist((size_t)maxdeg + 1, 0);
    for (int v = 0; v < n; ++v) ++hist[(size_t)deg[(size_t)v]];
    int64_t taken = 0, top = 0;
    for (int d = maxdeg; d >= 0 && taken < n / 10; --d) {
      const int64_t t = std::min<int64_t>(hist[(size_t)d], n / 10 - taken);
      taken += t;
      top += t * d;
    }
    if (2 * top < nnz) return TBSLA_OK;  // no hot set worth packing
  }
  // vertices by out-degree class, then in-degree, both descending: one stable
  // sort of (class, in-degree) keys
  const int grid = entry_grid(n), egrid = entry_grid(nnz);
  tbsla_matrix *B = new_matrix(TBSLA_FMT_CSR);
  if (!B) return fail(TBSLA_ERR_OOM, "host allocation failed");
  struct Guard {
    tbsla_matrix *B;
    int *newid = nullptr;
    ~Guard() {
      if (newid) cudaFree(newid);
      if (B) free_matrix(B);
    }
  } guard{B};
  B->device = A->device;
  TB_CUDA(cudaSetDevice(A->device));
  if (cudaMalloc(&guard.newid, (size_t)n * sizeof(int)) != cudaSuccess) {
    cudaGetLastError();
    return fail(TBSLA_ERR_OOM, "relabel map (%d ints)", n);
  }
  {
    SortScratch sc;
    SortPairs<uint64_t> p;
    TB_TRY(p.get(sc, n));
    const int top_cls = cls_max(maxdeg);
    vertex_keys_kernel<<<grid, 256>>>(d_deg, A->idx0, n, top_cls, p.keys, p.entries);
    TB_TRY(p.sort(sc, 32 + key_bits((uint64_t)top_cls)));
    new_labels_kernel<<<grid, 256>>>(p.entries, n, guard.newid);
    TB_CUDA(cudaGetLastError());
  }
  B->n_row = B->n_col = B->rows = n;
  B->stored = nnz;
  // columns with entries come first (their class is above that of degree 0)
  B->x_extent = n - std::count(deg.begin(), deg.end(), 0);
  TB_TRY(alloc_ints(B, &B->idx0, (int64_t)n + 1));
  // the entries by (new row, new column), repeated columns in their order: a
  // stable sort by column, then one by row
  SortScratch kept;
  int *order = nullptr;
  {
    SortScratch sc;
    SortPairs<uint32_t> p;
    TB_TRY(p.get(sc, nnz));
    const int bits = key_bits((uint64_t)std::max(n - 1, 0));
    new_column_keys_kernel<<<egrid, 256>>>(A->idx1, A->f_col, guard.newid, nnz, p.keys, p.entries);
    TB_TRY(p.sort(sc, bits));
    entry_rows_kernel<<<152 * 16, 256>>>(n, A->idx0, reinterpret_cast<int *>(p.other_keys));
    new_rows_kernel<<<egrid, 256>>>(guard.newid, nnz, p.other_keys);
    take_kernel<<<egrid, 256>>>(p.other_keys, p.entries, nnz, p.keys);
    TB_TRY(p.sort(sc, bits));
    key_starts_kernel<<<entry_grid((int64_t)n + 1), 256>>>(p.keys, nnz, (int64_t)n, B->idx0);
    TB_CUDA(cudaGetLastError());
    order = p.entries;
    sc.give(order);
    kept.owned.push_back(order);
  }
  TB_TRY(alloc_ints(B, &B->idx1, nnz));
  take_columns_kernel<<<egrid, 256>>>(A->idx1, A->f_col, guard.newid, order, nnz, B->idx1);
  TB_TRY(take_values(B, A, order));
  TB_CUDA(cudaStreamSynchronize(0));
  kept.drop(order);
  std::vector<int> nrp((size_t)n + 1), newid((size_t)n);
  TB_CUDA(cudaMemcpy(nrp.data(), B->idx0, nrp.size() * sizeof(int), cudaMemcpyDeviceToHost));
  TB_CUDA(cudaMemcpy(newid.data(), guard.newid, newid.size() * sizeof(int), cudaMemcpyDeviceToHost));
  TB_TRY(csr_bins(B, nrp));
  int *d_newid = guard.newid;
  guard.newid = nullptr;
  guard.B = nullptr;
  B->x_keep = A->x_keep;
  B->x_keep_range = A->x_keep_range;
  B->short_mode = A->short_mode;
  B->pr_polls = A->pr_polls;
  A->pr_relabel = B;
  A->pr_newid = d_newid;
  A->pr_newid_host = std::move(newid);
  *built = true;
  return TBSLA_OK;
}

}  // namespace

// The relabelled copy to run PageRank on, or NULL for A itself.
tbsla_status_t pr_relabelled(tbsla_matrix *A, tbsla_matrix **B) {
  *B = nullptr;
  if (A->pr_relabel_mode == 0 || !candidate(A)) return TBSLA_OK;
  std::lock_guard<std::mutex> lk(A->first_use);
  if (A->pr_relabel_state == 1) {
    *B = A->pr_relabel;
    return TBSLA_OK;
  }
  if (A->pr_relabel_state == 2 && A->pr_relabel_mode == -1) return TBSLA_OK;
  const bool forced = A->pr_relabel_mode == 1;
  if (!forced) {
    bool is_banded = true;
    if (A->n_row < (1 << 20)) {
      A->pr_relabel_state = 2;
      return TBSLA_OK;
    }
    TB_TRY(banded(A, &is_banded));
    if (is_banded) {
      A->pr_relabel_state = 2;
      return TBSLA_OK;
    }
  }
  // the copy only makes the solve faster: without the device memory for it
  // (16 bytes an entry to sort, then the copy) A itself is swept, and unless the copy
  // was asked for the build is not tried again until the values change
  bool built = false;
  const tbsla_status_t st = build(A, !forced, &built);
  if (st == TBSLA_ERR_OOM) forget_error();
  else TB_TRY(st);
  A->pr_relabel_state = built ? 1 : 2;
  *B = built ? A->pr_relabel : nullptr;
  return TBSLA_OK;
}

}  // namespace tbsla
