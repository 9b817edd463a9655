// device_sort.cuh -- the entries of a CSR handle in another order, on the
// device: stable radix sorts of (key, entry) pairs (CUB, as the conversions
// use) and the kernels around them.  Shared by the transposed copy and the
// degree-relabelled PageRank copy, which a handle builds on first use; sorting
// and copying the entries on the host took 175 ms for 16.8 million of them
// (transposed) and half a second for 31 million (relabelled).
#pragma once

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>
#include <algorithm>
#include <vector>

#include "common.cuh"

namespace tbsla {

tbsla_matrix *new_matrix(int format);
void free_matrix(tbsla_matrix *A);
tbsla_status_t alloc_ints(tbsla_matrix *A, int **p, int64_t n);
tbsla_status_t rederive_stores(tbsla_matrix *A, cudaStream_t s);
tbsla_status_t csr_bins(tbsla_matrix *A, const std::vector<int> &rp);

// Device scratch: freed together at the end, or one by one as soon as it is not
// needed (cudaFree waits for the device)
struct SortScratch {
  std::vector<void *> owned;
  ~SortScratch() {
    for (void *p : owned) cudaFree(p);
  }
  template <typename T> tbsla_status_t get(T **p, int64_t n) {
    void *q = nullptr;
    if (cudaMalloc(&q, (size_t)std::max<int64_t>(n, 1) * sizeof(T) + 64) != cudaSuccess) {
      cudaGetLastError();
      return fail(TBSLA_ERR_OOM, "sort scratch (%lld bytes)", (long long)(n * (int64_t)sizeof(T)));
    }
    owned.push_back(q);
    *p = static_cast<T *>(q);
    return TBSLA_OK;
  }
  // p belongs to the caller from here on
  void give(void *p) { owned.erase(std::find(owned.begin(), owned.end(), p)); }
  void drop(void *p) {
    give(p);
    cudaFree(p);
  }
};

inline int key_bits(uint64_t largest) {
  int b = 1;
  while (b < 64 && (largest >> b)) ++b;
  return b;
}

// The keys and entries of a sort and the second pair of arrays it needs: 16 bytes
// an entry with 32-bit keys, as much as a plain FP64 copy and its map take
// afterwards, so that a copy which fits can also be built
template <typename K> struct SortPairs {
  K *keys = nullptr, *other_keys = nullptr;
  int *entries = nullptr, *other_entries = nullptr;
  int64_t n = 0;
  tbsla_status_t get(SortScratch &sc, int64_t n_) {
    n = n_;
    TB_TRY(sc.get(&keys, n));
    TB_TRY(sc.get(&other_keys, n));
    TB_TRY(sc.get(&entries, n));
    return sc.get(&other_entries, n);
  }
  // into increasing key order, equal keys as they were
  tbsla_status_t sort(SortScratch &sc, int bits) {
    cub::DoubleBuffer<K> kb(keys, other_keys);
    cub::DoubleBuffer<int> eb(entries, other_entries);
    size_t bytes = 0;
    TB_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, bytes, kb, eb, n, 0, bits));
    char *tmp = nullptr;
    TB_TRY(sc.get(&tmp, (int64_t)bytes));
    TB_CUDA(cub::DeviceRadixSort::SortPairs(tmp, bytes, kb, eb, n, 0, bits));
    sc.drop(tmp);
    keys = kb.Current();
    other_keys = kb.Alternate();
    entries = eb.Current();
    other_entries = eb.Alternate();
    return TBSLA_OK;
  }
};

namespace {

// row of every entry: a warp per row
__global__ void __launch_bounds__(256) entry_rows_kernel(int rows, const int *__restrict__ rowptr,
                                                        int *__restrict__ row) {
  const int lane = threadIdx.x & 31;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < rows; r += nw)
    for (int k = __ldg(rowptr + r) + lane; k < __ldg(rowptr + r + 1); k += 32) row[k] = (int)r;
}

// begin[j] = the first position whose key is at least j, j <= count
template <typename K>
__global__ void __launch_bounds__(256) key_starts_kernel(const K *__restrict__ sorted, int64_t n, int64_t count,
                                                        int *__restrict__ begin) {
  for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j <= count; j += (int64_t)gridDim.x * blockDim.x) {
    int64_t lo = 0, hi = n;
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if ((int64_t)sorted[mid] < j) lo = mid + 1;
      else hi = mid;
    }
    begin[j] = (int)lo;
  }
}

template <typename T>
__global__ void __launch_bounds__(256) take_kernel(const T *__restrict__ src, const int *__restrict__ order, int64_t n,
                                                  T *__restrict__ out) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x)
    out[k] = src[order[k]];
}

inline int entry_grid(int64_t n) { return (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 152 * 32)); }

// The stores of B, those that A has (F64 among them), from A's values in another order
inline tbsla_status_t take_values(tbsla_matrix *B, const tbsla_matrix *A, const int *order) {
  const int64_t n = A->stored;
  const size_t size[3] = {8, 4, 2};
  for (int k = 0; k < 3; ++k)
    if (A->values[k]) TB_TRY(dev_alloc(B, &B->values[k], (size_t)n * size[k]));
  B->stores = A->stores;
  if (n)
    take_kernel<<<entry_grid(n), 256>>>(static_cast<const double *>(A->values[0]), order, n,
                                        static_cast<double *>(B->values[0]));
  TB_CUDA(cudaGetLastError());
  return rederive_stores(B, 0);
}

}  // namespace
}  // namespace tbsla
