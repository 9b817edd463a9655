// pagerank.cu -- PageRank on GB300: fused sweeps, deterministic reductions, FP64
// and mixed precision.
//
// A sweep is one SpMV whose epilogue writes the new iterate and accumulates
// partial sums (residual, dangling mass, total mass, or the maximum; with
// acceleration the residual dots); all sweeps of a solve run in one
// cooperative launch (pr_sweep.cuh) for the layouts it walks: CSR and
// row-sorted COO row items, the ELL layout.  Others (DENSE, rows the format
// never visits) launch their product and one step of
// the same kernel per sweep.  No atomics on values: every result is
// independent of scheduling.
//
// Modes
//   TBSLA_PR_REFERENCE  Matrix::page_rank (src/cpp/matrix/Matrix.cpp:13-61):
//     b = beta*A b_prev + (1-beta)/n * sum(b_prev); b /= max(b);
//     err = sum |b - b_prev|; finally b /= sum(b).  With a node list this is
//     Matrix::personalized_page_rank (Matrix.cpp:63-114).
//   TBSLA_PR_DANGLING   x = beta*A x + (beta*dangling(x) + (1-beta)*sum(x))/n,
//     stop when ||x - x_prev||_1 < tol.
//   accelerated (DANGLING, FP64, accel = 1): Anderson acceleration of the
//     same fixed-point map over the last two differences, same stopping rule
//     on ||G(x) - x||_1, the result is G(x) of the last sweep.
//   mixed precision (DANGLING, precision F32/BF16): FP64 defect correction.
//     r = G(x) - x by an FP64 sweep (its L1 norm is the stopping quantity),
//     then e_{j+1} = G~ e_j + r by sweeps on the reduced-precision value store
//     with FP32 vectors until ||e_{j+1} - e_j||_1 < inner_tol, x += e (FP64).
//     The FP64 sweep and the correction solve are one launch each, queued
//     without waiting for the host.
#include <climits>
#include <cmath>
#include <cstring>
#include <vector>

#include "column_mask.cuh"
#include "pr_sweep.cuh"
#include "product.cuh"

namespace tbsla {

tbsla_status_t spmv_dispatch(const tbsla_matrix *A, tbsla_dtype_t store, tbsla_dtype_t xt, const void *x,
                             tbsla_dtype_t yt, void *y, int vect_incr, cudaStream_t s);

namespace {

// out = (beta * mass + 1 - beta) * x with mass = the sum of the partials
__global__ void __launch_bounds__(256) pr_mass_kernel(const double *__restrict__ v, int n,
                                                      const unsigned char *__restrict__ dmask, double *partials) {
  __shared__ double sh[256];
  double d = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    if (dmask[i]) d += v[i];
  const double t = block_sum<256, double>(d, sh);
  if (threadIdx.x == 0) partials[blockIdx.x] = t;
}
__global__ void __launch_bounds__(256) pr_scale_to_kernel(const double *__restrict__ x, int n,
                                                          const double *__restrict__ partials, int nparts,
                                                          double beta, double *__restrict__ out) {
  __shared__ double sh[256];
  __shared__ double mass;
  double d = 0;
  for (int k = threadIdx.x; k < nparts; k += 256) d += partials[k];
  const double t = block_sum<256, double>(d, sh);
  if (threadIdx.x == 0) mass = t;
  __syncthreads();
  const double f = beta * mass + (1.0 - beta);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) out[i] = f * x[i];
}

__global__ void pr_dangling_dense_kernel(const double *__restrict__ a, int rows, int cols, unsigned char *dmask) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < cols; j += gridDim.x * blockDim.x) {
    bool any = false;
    for (int i = 0; i < rows && !any; ++i) any = a[(size_t)i * cols + j] != 0.0;
    if (any) dmask[j] = 0;
  }
}


// ------------------------------------------------------------ workspace
constexpr int kMassBlocks = 152 * 2;
// the control block and, after it, the grid barrier's words
constexpr size_t kCtlBytes = (sizeof(PrCtl) + 127) / 128 * 128;
constexpr size_t kBarBytes = kPrBarWords * sizeof(unsigned);

struct PrWork {
  int n = 0;
  double *x[2] = {nullptr, nullptr};  // FP64 iterates
  double *prod = nullptr;             // plain product (layouts the solver does not walk)
  float *e[2] = {nullptr, nullptr};   // inner iterates
  float *prod32 = nullptr;
  float *r = nullptr;
  unsigned char *dmask = nullptr, *tmask = nullptr;
  double *lam = nullptr;              // adjoint solution
  double *ag[3] = {nullptr, nullptr, nullptr};  // accelerated solve: sweep outputs (slot k % 3)
  double *ar[3] = {nullptr, nullptr, nullptr};  // and their residuals
  float *eg[3] = {nullptr, nullptr, nullptr};   // accelerated inner solve: outputs (slot k % 3)
  float *er[3] = {nullptr, nullptr, nullptr};   // and their residuals
  double *partials = nullptr;
  int part_stride = 0;
  PrCtl *ctl = nullptr;
  unsigned *bar = nullptr;            // grid barrier, in ctl's allocation
  PrCtl *ctl_host = nullptr;          // pinned copy of both
  cudaStream_t stream = nullptr;
  ~PrWork() {
    void *ps[] = {x[0], x[1], prod, e[0], e[1], prod32, r, dmask, tmask, lam, partials, ctl,
                  ag[0], ag[1], ag[2], ar[0], ar[1], ar[2], eg[0], eg[1], eg[2], er[0], er[1], er[2]};
    for (void *p : ps) if (p) cudaFree(p);
    if (ctl_host) cudaFreeHost(ctl_host);
    if (stream) cudaStreamDestroy(stream);
  }
};

tbsla_status_t pr_alloc(void **p, size_t bytes) {
  const cudaError_t e = cudaMalloc(p, bytes + 64);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(TBSLA_ERR_OOM, "cudaMalloc(%zu) for PageRank failed: %s", bytes, cudaGetErrorString(e));
  }
  return TBSLA_OK;
}

// ------------------------------------------------------------ plan
// The layouts the solver kernel walks itself, every row visited exactly once.  The
// kernel variant of the handle's products makes no difference: the row pointer
// and the slots are there for all of them, and a product and a step per sweep
// cost more launches than the graph of sweeps that such handles had (row-sorted
// COO with the merge path, 65536 rows, 17 sweeps: 757 us, 626 as a graph, 246
// walked; ELL with four rows a thread, 16 sweeps: 410, 343, 243).
bool walks_items(const tbsla_matrix *A) {
  const bool csr = A->format == TBSLA_FMT_CSR;
  const bool coo = (A->format == TBSLA_FMT_COO || A->format == TBSLA_FMT_SCOO) && A->coo_rowptr;
  return (csr || coo) && A->rows == A->n_row && A->stored > 0 && A->stored <= INT_MAX - 4096;
}
bool walks_slots(const tbsla_matrix *A) {
  return A->format == TBSLA_FMT_ELL && A->rows == A->n_row && A->rows > 0 && A->max_col > 0;
}

// cnt[0] of cnt[1] entries of sampled rows have the entry at their place in the next
// row within kNearCols columns of it (a warp per sampled row)
constexpr int kNearSamples = 4096, kNearCols = 1024;
__global__ void __launch_bounds__(256) near_columns_kernel(const int *__restrict__ rowptr, const int *__restrict__ colidx,
                                                          int rows, unsigned long long *cnt) {
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  const int r = (int)((int64_t)w * (rows - 1) / kNearSamples);
  const int a = rowptr[r], b = rowptr[r + 1], len = min(b - a, rowptr[r + 2] - b);
  unsigned near = 0;
  for (int k = lane; k < len; k += 32) near += abs(colidx[a + k] - colidx[b + k]) <= kNearCols;
  near = __reduce_add_sync(0xffffffffu, near);
  if (lane == 0 && len > 0) {
    atomicAdd(cnt, (unsigned long long)near);
    atomicAdd(cnt + 1, (unsigned long long)len);
  }
}

// Whether neighbouring rows of A (row items) gather neighbouring entries of the
// iterate; the pattern's, kept with the handle
tbsla_status_t near_columns(tbsla_matrix *A, bool *near) {
  if (!A->pr_near) {
    unsigned long long *d = nullptr, h[2] = {0, 0};
    if (A->rows >= 2) {
      TB_TRY(pr_alloc((void **)&d, sizeof h));
      cudaError_t e = cudaMemset(d, 0, sizeof h);
      if (e == cudaSuccess)
        near_columns_kernel<<<kNearSamples * 32 / 256, 256>>>(A->format == TBSLA_FMT_CSR ? A->idx0 : A->coo_rowptr,
                                                              A->idx1, A->rows, d);
      if (e == cudaSuccess) e = cudaMemcpy(h, d, sizeof h, cudaMemcpyDeviceToHost);
      cudaFree(d);
      TB_CUDA(e);
    }
    A->pr_near = h[1] && 2 * h[0] >= h[1] ? 1 : 2;
  }
  *near = A->pr_near == 1;
  return TBSLA_OK;
}

struct PlanHolder {
  PrPlan p;
  ~PlanHolder() {
    void *ps[] = {p.items, p.empty, p.chunks, p.arrived, p.partial};
    for (void *q : ps) if (q) cudaFree(q);
  }
};

// The row classes of the solver (PrPlan).  `share` is a thread's part of the
// entries.  Large graphs: one lane a row of at most four entries (one batch),
// 4 lanes up to 64, 8 up to 256, 32 up to half a lane's share of the sweep,
// then chunks of eight warps: long walks by few lanes cost the fewest
// reduction steps, but no row may outlast the sweep.  Where rows of up to 16
// entries (32, if nine tenths of the entries lie in such rows) hold half of
// the entries, and neighbouring rows gather neighbouring entries or the rows are
// short (of those above four entries, fewer than 10 on average), they take one
// lane with 16-byte loads instead of four: the gathers hit L1 or L2 then, and four
// lanes a row cost instructions, FP64 additions above all (cqmat, 2^22 rows of
// 8, BF16: 13.1 ms with four lanes, 7.2 so; its adjoint 4.9 and 3.4; 2^22 random
// rows of 6 on average, FP64: 4.5 and 3.8).  Random gathers of longer rows need the
// four lanes' loads in flight (2^20 rows of 12, FP32: 1.60 ms, one lane 1.75).
// Small graphs, where a warp takes an item or two a sweep: one lane up to 8, 4 up
// to 32, 8 up to 128, 32 up to 512 entries, four batches at most (FP64 training
// step on R-MAT 2^16 / 2^13: 1743 / 1384 us; half as long 1920 / 1546; FP32
// solve on 2^18 752 against 813).  Depends on the pattern only: kept with the
// handle across value changes.
tbsla_status_t solver_plan(tbsla_matrix *A, const PrPlan **out) {
  if (A->pr_plan) {
    *out = &static_cast<PlanHolder *>(A->pr_plan)->p;
    return TBSLA_OK;
  }
  const int rows = A->rows;
  std::vector<int> rp((size_t)rows + 1);
  TB_CUDA(cudaMemcpy(rp.data(), A->format == TBSLA_FMT_CSR ? A->idx0 : A->coo_rowptr, rp.size() * sizeof(int),
                     cudaMemcpyDeviceToHost));
  const int64_t share = A->stored / (152 * kPrThreads);
  const int per = (int)std::max<int64_t>(16, std::min<int64_t>(share / 2, 128));
  const bool small = share < 32;
  // wide items: rows of 5 to `wide` entries (none: wide = one)
  const int one = small ? 8 : 4;
  int wide = one;
  if (!small) {
    int64_t entries[2] = {0, 0}, count[2] = {0, 0};  // of rows up to 16, up to 32
    int64_t upto32 = 0;
    for (int r = 0; r < rows; ++r) {
      const int len = rp[(size_t)r + 1] - rp[(size_t)r];
      if (len > 32) continue;
      upto32 += len;
      for (int k = 0; k < 2; ++k)
        if (len > one && len <= 16 << k) {
          entries[k] += len;
          ++count[k];
        }
    }
    const int k = 10 * upto32 >= 9 * A->stored;
    bool take = false;
    if (2 * entries[k] >= A->stored) {
      take = entries[k] < 10 * count[k];
      if (!take) TB_TRY(near_columns(A, &take));
    }
    if (take) wide = 16 << k;
  }
  // longest row of 32, 8 and 4 lanes, a wide one, one of one lane, and a chunk
  const int limit[5] = {32 * per, small ? 128 : 256, small ? 32 : 64, wide, one}, chunk = kPrSub * std::min(per, 32);
  std::vector<int4> chunk_items, chunks;
  int count[5] = {0, 0, 0, 0, 0};
  auto bucket = [&](int len) { return len > limit[1] ? 0 : len > limit[2] ? 1 : len > limit[3] ? 2 : len > limit[4] ? 3 : 4; };
  int n_empty = 0;
  for (int r = 0; r < rows; ++r) {
    const int len = rp[(size_t)r + 1] - rp[(size_t)r];
    if (len == 0) ++n_empty;
    else if (len <= limit[0]) ++count[bucket(len)];
  }
  int at[5], first[5], total = 0;
  for (int b = 0; b < 5; ++b) {
    first[b] = at[b] = total;
    total += count[b];
  }
  PlanHolder *H = new PlanHolder;
  PrPlan &p = H->p;
  std::vector<int4> items((size_t)total);
  std::vector<int> empty((size_t)n_empty);
  n_empty = 0;
  for (int r = 0; r < rows; ++r) {
    const int a = rp[(size_t)r], b = rp[(size_t)r + 1], len = b - a;
    if (len == 0) {
      empty[(size_t)n_empty++] = r;
    } else if (len <= limit[0]) {
      items[(size_t)at[bucket(len)]++] = make_int4(r, a, b, -1);
    } else if (len <= chunk) {
      chunk_items.push_back(make_int4(r, a, b, -1));
    } else {
      const int slot = (int)chunks.size(), n = (len + chunk - 1) / chunk;
      for (int c = 0; c < n; ++c) {
        chunk_items.push_back(make_int4(r, a + c * chunk, std::min(b, a + (c + 1) * chunk), slot + c));
        chunks.push_back(make_int4(r, slot, n, p.n_chunked));
      }
      ++p.n_chunked;
    }
  }
  const int nc = (int)chunk_items.size();
  p.start[0] = 0;
  p.start[1] = nc;
  p.start[2] = nc + first[1];
  p.start[3] = nc + first[2];
  p.start[4] = nc + first[4];  // wide items are the last of the 4-lane class
  p.start[5] = nc + total;
  p.n_wide = count[3];
  p.n_empty = n_empty;
  p.slots = (int)chunks.size();
  chunk_items.insert(chunk_items.end(), items.begin(), items.end());
  tbsla_status_t st = TBSLA_OK;
  auto put = [&](void **d, const void *h, size_t bytes) {
    if (st == TBSLA_OK) st = pr_alloc(d, bytes);
    if (st == TBSLA_OK && bytes &&
        (h ? cudaMemcpy(*d, h, bytes, cudaMemcpyHostToDevice) : cudaMemset(*d, 0, bytes)) != cudaSuccess)
      st = fail(TBSLA_ERR_CUDA, "PageRank work list upload");
  };
  put((void **)&p.items, chunk_items.data(), chunk_items.size() * sizeof(int4));
  put((void **)&p.empty, empty.data(), empty.size() * sizeof(int));
  put((void **)&p.chunks, chunks.data(), chunks.size() * sizeof(int4));
  put((void **)&p.arrived, nullptr, (size_t)p.n_chunked * sizeof(int));
  put((void **)&p.partial, nullptr, (size_t)p.slots * sizeof(double));
  if (st != TBSLA_OK) {
    delete H;
    return st;
  }
  A->pr_plan = H;
  A->pr_plan_free = [](void *q) { delete static_cast<PlanHolder *>(q); };
  *out = &p;
  return TBSLA_OK;
}

// What the solver sweeps for the value store `vals` of A: where it walks A itself
// the ELL layout (an ELL handle, or the copy of a CSR / COO handle) or the row
// items, else a product launched before each step.
template <typename V, typename T>
tbsla_status_t solver_matrix(tbsla_matrix *A, const V *vals, bool walked, T *prod, PrMat<V, T> *m) {
  std::memset(m, 0, sizeof *m);
  m->rows = A->n_row;
  m->f_col = A->f_col;
  m->prod = prod;
  m->layout = kPrProduct;
  if (!walked) return TBSLA_OK;
  if (walks_slots(A)) {
    m->layout = kPrSlots;
    m->ecols = A->idx0;
    m->evals = vals;
    m->estride = A->rows_pad;
    m->ewidth = A->max_col;
  } else {
    const void *copy = nullptr;
    for (int k = 0; k < 2; ++k)
      if (A->sell_width && A->values[k] == static_cast<const void *>(vals)) copy = A->sell_vals[k];
    if (copy && (A->short_mode == -1 || A->short_mode == 3)) {
      m->layout = kPrSlots;
      m->ecols = A->sell_cols;
      m->evals = static_cast<const V *>(copy);
      m->estride = A->sell_stride;
      m->ewidth = A->sell_width;
    } else {
      const PrPlan *p = nullptr;
      TB_TRY(solver_plan(A, &p));
      m->layout = kPrItems;
      m->plan = *p;
      m->colidx = A->idx1;
      m->values = vals;
    }
  }
  return TBSLA_OK;
}

// Largest sweep count of one launch: launches of at most about a second, so
// that the host sees the control block now and then
int sweep_limit(const tbsla_matrix *A) {
  const double work = (double)A->stored + 8.0 * A->n_row + 1e6;
  return (int)std::max(16.0, std::min(1e6, 2e11 / work));
}

// Polls of a grid barrier before a block gives up: more than a second's worth,
// and more than the longest wait in the order of things, for a lane that walks
// an ELL row (up to half a microsecond a slot where the row is nearly alone on
// its SM, at least a tenth a poll)
template <typename V, typename T> unsigned barrier_polls(const tbsla_matrix *A, const PrMat<V, T> &m) {
  if (A->pr_polls) return A->pr_polls;
  const int64_t slots = m.layout == kPrSlots ? m.ewidth : 0;
  return (unsigned)std::min<int64_t>((1 << 22) + 16 * slots, 1u << 31);
}

constexpr int kRefProductRows = 1 << 22;

template <bool kWide, int MODE, typename V, typename T, bool AA>
tbsla_status_t launch_kind(const tbsla_matrix *A, const PrMat<V, T> &m, PrArgs<T> &a, const PrWork *W,
                           cudaStream_t s) {
  static int per_sm[64], sms[64];
  static std::once_flag once[64];
  const int dev = A->device < 64 ? A->device : 63;
  std::call_once(once[dev], [&] {
    cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, A->device);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm[dev], pr_solve_kernel<kWide, MODE, V, T, AA>, kPrThreads, 0);
  });
  TB_CHECK(per_sm[dev] > 0, "the PageRank solver does not fit on the device");
  // four entries or one row per thread, all blocks resident at once
  const int64_t want = ((int64_t)A->stored / 4 + A->n_row + kPrThreads - 1) / kPrThreads;
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(want, (int64_t)sms[dev] * per_sm[dev]));
  a.partials = W->partials;
  a.part_stride = W->part_stride;
  a.n = W->n;
  a.ctl = W->ctl;
  a.bar = W->bar;
  a.polls = barrier_polls(A, m);
  TB_CHECK(grid + (m.layout == kPrItems ? m.plan.n_chunked : 0) <= W->part_stride, "PageRank partials too small");
  void *args[] = {const_cast<PrMat<V, T> *>(&m), &a};
  TB_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(pr_solve_kernel<kWide, MODE, V, T, AA>), dim3(grid),
                                      dim3(kPrThreads), args, 0, s));
  return TBSLA_OK;
}

template <int MODE, typename V, typename T, bool AA>
tbsla_status_t launch_solver(const tbsla_matrix *A, const PrMat<V, T> &m, PrArgs<T> &a, const PrWork *W,
                             cudaStream_t s) {
  if (m.layout == kPrItems && m.plan.n_wide > 0) return launch_kind<true, MODE, V, T, AA>(A, m, a, W, s);
  return launch_kind<false, MODE, V, T, AA>(A, m, a, W, s);
}

// the partials: one slot per block of a full grid and per chunked row
constexpr int kPrGridMax = 512;
tbsla_status_t pr_partials(PrWork *W, int chunked) {
  const int need = kPrGridMax + chunked;
  if (W->part_stride >= need) return TBSLA_OK;
  if (W->partials) cudaFree(W->partials);
  W->partials = nullptr;
  W->part_stride = 0;
  TB_TRY(pr_alloc((void **)&W->partials, (size_t)need * 2 * 6 * 8));
  W->part_stride = need;
  return TBSLA_OK;
}

// dangling columns: those without a nonzero stored value
tbsla_status_t pr_dangling_mask(tbsla_matrix *A, PrWork *W) {
  const int n = W->n, g = 152 * 8;
  TB_CUDA(cudaMemsetAsync(W->dmask, 1, (size_t)n, W->stream));
  switch (A->format) {
  case TBSLA_FMT_CSR:
  case TBSLA_FMT_COO:
  case TBSLA_FMT_SCOO: {
    int *zeros = reinterpret_cast<int *>(W->bar) + kPrBarWords;
    if (A->values[0]) TB_TRY(column_mask(A, (const double *)A->values[0], W->dmask, zeros, W->stream));
    else if (A->values[1]) TB_TRY(column_mask(A, (const float *)A->values[1], W->dmask, zeros, W->stream));
    break;
  }
  case TBSLA_FMT_ELL:
    if (A->values[0])
      column_mark_kernel<double><<<g, 256, 0, W->stream>>>(A->idx0, (const double *)A->values[0],
                                                           (int64_t)A->rows_pad * A->max_col, A->f_col, n, nullptr,
                                                           W->dmask);
    break;
  case TBSLA_FMT_DENSE:
    if (A->values[0]) pr_dangling_dense_kernel<<<g, 256, 0, W->stream>>>((const double *)A->values[0], A->rows, A->cols, W->dmask);
    break;
  }
  TB_CUDA(cudaGetLastError());
  return TBSLA_OK;
}

tbsla_status_t pr_setup(tbsla_matrix *A, PrWork **out) {
  PrWork *W = static_cast<PrWork *>(A->pr_work);
  if (!W) {
    W = new PrWork();
    const int n = A->n_col;
    W->n = n;
    tbsla_status_t st = TBSLA_OK;
    auto alloc = [&](void **p, size_t b) { if (st == TBSLA_OK) st = pr_alloc(p, b); };
    alloc((void **)&W->x[0], (size_t)n * 8);
    alloc((void **)&W->x[1], (size_t)n * 8);
    alloc((void **)&W->dmask, (size_t)n);
    alloc((void **)&W->tmask, (size_t)n);
    alloc((void **)&W->ctl, kCtlBytes + kBarBytes + sizeof(int));  // and the mask's scratch
    W->bar = reinterpret_cast<unsigned *>(reinterpret_cast<char *>(W->ctl) + kCtlBytes);
    if (st == TBSLA_OK && cudaMallocHost((void **)&W->ctl_host, kCtlBytes + kBarBytes) != cudaSuccess)
      st = fail(TBSLA_ERR_OOM, "pinned control block");
    if (st == TBSLA_OK && cudaStreamCreateWithFlags(&W->stream, cudaStreamNonBlocking) != cudaSuccess)
      st = fail(TBSLA_ERR_CUDA, "stream creation failed");
    if (st == TBSLA_OK && cudaMemsetAsync(W->bar, 0, kBarBytes, W->stream) != cudaSuccess)
      st = fail(TBSLA_ERR_CUDA, "PageRank setup");
    if (st != TBSLA_OK) { delete W; return st; }
    A->pr_work = W;
    A->pr_work_free = [](void *p) { delete static_cast<PrWork *>(p); };
    A->pr_dmask_stale = true;
  }
  if (A->pr_dmask_stale) {
    TB_TRY(pr_dangling_mask(A, W));
    A->pr_dmask_stale = false;
  }
  *out = W;
  return TBSLA_OK;
}

tbsla_status_t pr_inner_buffers(PrWork *W, bool accel) {
  const size_t b = (size_t)W->n * 4;
  if (!W->r) {
    TB_TRY(pr_alloc((void **)&W->e[0], b));
    TB_TRY(pr_alloc((void **)&W->e[1], b));
    TB_TRY(pr_alloc((void **)&W->r, b));
  }
  if (accel && !W->er[2])
    for (int i = 0; i < 3; ++i) {
      if (!W->eg[i]) TB_TRY(pr_alloc((void **)&W->eg[i], b));
      if (!W->er[i]) TB_TRY(pr_alloc((void **)&W->er[i], b));
    }
  return TBSLA_OK;
}

// the ring buffers of the accelerated solves
tbsla_status_t pr_aa_buffers(PrWork *W) {
  if (W->ar[2]) return TBSLA_OK;
  for (int i = 0; i < 3; ++i) {
    if (!W->ag[i]) TB_TRY(pr_alloc((void **)&W->ag[i], (size_t)W->n * 8));
    if (!W->ar[i]) TB_TRY(pr_alloc((void **)&W->ar[i], (size_t)W->n * 8));
  }
  return TBSLA_OK;
}

// Waits for the solve's stream.  A barrier that was given up leaves the blocks
// in different sweeps: the barrier and the chunk counts of the swept matrix's
// plan (blocks that went on have counted chunks the others never did) are reset
// for the next solve, and the error is returned.
tbsla_status_t pr_wait(const tbsla_matrix *A, PrWork *W) {
  TB_CUDA(cudaGetLastError());
  TB_CUDA(cudaMemcpyAsync(W->ctl_host, W->ctl, kCtlBytes + kBarBytes, cudaMemcpyDeviceToHost, W->stream));
  TB_CUDA(cudaStreamSynchronize(W->stream));
  const unsigned *bar = reinterpret_cast<const unsigned *>(reinterpret_cast<const char *>(W->ctl_host) + kCtlBytes);
  if (bar[kPrGaveUp]) {
    TB_CUDA(cudaMemsetAsync(W->bar, 0, kBarBytes, W->stream));
    if (A->pr_plan) {
      const PrPlan &p = static_cast<const PlanHolder *>(A->pr_plan)->p;
      TB_CUDA(cudaMemsetAsync(p.arrived, 0, (size_t)p.n_chunked * sizeof(int), W->stream));
    }
    TB_CUDA(cudaStreamSynchronize(W->stream));
    return fail(TBSLA_ERR_TIMEOUT, "a grid barrier of the PageRank solver ran out of polls");
  }
  return TBSLA_OK;
}

// The solve's stream waits for the work queued on the caller's stream (NULL: the
// legacy stream, with which a non-blocking stream has no order of its own):
// teleport vectors and incoming gradients may still be written there, and the
// result's buffer still read.
tbsla_status_t pr_order(PrWork *W, cudaStream_t user) {
  cudaEvent_t ev;
  TB_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
  cudaError_t e = cudaEventRecord(ev, user);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(W->stream, ev, 0);
  cudaEventDestroy(ev);
  TB_CUDA(e);
  return TBSLA_OK;
}

// kernel timing records events around products; none inside a solve
struct TimingOff {
  tbsla_matrix *A;
  bool was;
  explicit TimingOff(tbsla_matrix *A_) : A(A_), was(A_->timing) { A->timing = false; }
  ~TimingOff() { A->timing = was; }
};

// The FP64 solve of one mode (args: its vectors and control block), result in args.out.
template <int MODE, bool AA>
tbsla_status_t run_f64(tbsla_matrix *A, PrWork *W, PrArgs<double> &a, int check_every) {
  if (AA) {
    TB_TRY(pr_aa_buffers(W));
    for (int i = 0; i < 3; ++i) {
      a.g[i] = W->ag[i];
      a.r[i] = W->ar[i];
    }
  }
  bool walked = walks_items(A) || walks_slots(A);
  // The reference mode never runs on the relabelled copy: on large graphs in
  // their own labels the gathers go to DRAM, and the plain product, with twice
  // the warps per SM, is faster by more than its launch and the step cost.  R-MAT
  // of 2^20 / 2^21 / 2^22 / 2^23 / 2^24 vertices, 16 sweeps: walked 1.8 / 4.0 /
  // 9.0 / 22.2 / 48.0 ms, by products 2.2 / 4.1 / 7.7 / 15.4 / 29.8; 2^22 random
  // rows of 3 / 16 / 48 entries, 20 sweeps: 5.1 / 15.3 / 28.4 and 4.1 / 10.3 / 25.9.
  // Where neighbouring rows gather neighbouring entries it is better walked at every
  // size (2^22 banded rows of 8 / 24: 5.5 / 7.9 ms, 8.6 / 11.0 by products), as the
  // ELL layout is (even rows; 2^24 of them, 205 sweeps: 118, 130 ms).
  if (MODE == kSweepRef && A->n_row >= kRefProductRows && walked && !walks_slots(A) &&
      !(A->sell_width && A->values[0] && (A->short_mode == -1 || A->short_mode == 3)))
    TB_TRY(near_columns(A, &walked));
  if (!walked && !W->prod) TB_TRY(pr_alloc((void **)&W->prod, (size_t)W->n * 8));
  PrMat<double, double> m;
  TB_TRY((solver_matrix<double, double>(A, static_cast<const double *>(A->values[0]), walked, W->prod, &m)));
  TB_TRY(pr_partials(W, m.layout == kPrItems ? m.plan.n_chunked : 0));
  a.x[0] = W->x[0];
  a.x[1] = W->x[1];
  a.init = 1;
  if (m.layout != kPrProduct) {
    a.limit = sweep_limit(A);
    do {
      TB_TRY((launch_solver<MODE, double, double, AA>(A, m, a, W, W->stream)));
      TB_TRY(pr_wait(A, W));
      a.init = 0;
    } while (!W->ctl_host->done);
    return TBSLA_OK;
  }
  a.limit = 0;
  TB_TRY((launch_solver<MODE, double, double, AA>(A, m, a, W, W->stream)));
  a.init = 0;
  a.limit = 1;
  int k = 0;
  do {
    for (int j = 0; j < check_every; ++j, ++k) {
      TB_TRY(spmv_dispatch(A, TBSLA_F64, TBSLA_F64, AA ? W->x[0] : W->x[k & 1], TBSLA_F64, W->prod, 0, W->stream));
      TB_TRY((launch_solver<MODE, double, double, AA>(A, m, a, W, W->stream)));
    }
    TB_TRY(pr_wait(A, W));
  } while (!W->ctl_host->done);
  return TBSLA_OK;
}

constexpr int kInnerMax = 512;  // sweeps of one correction solve at most

// The mixed-precision solve (dangling mode): an FP64 sweep for r = G(x) - x,
// the correction solve on the value store V, x += e, queued without waiting
// (launches after the last sweep return at once).
template <typename V, bool AA>
tbsla_status_t run_mixed(tbsla_matrix *A, PrWork *W, PrArgs<double> &a, tbsla_dtype_t store, int check_every) {
  TB_TRY(pr_inner_buffers(W, AA));
  const bool walked = walks_items(A) || walks_slots(A);
  if (!walked && !W->prod) TB_TRY(pr_alloc((void **)&W->prod, (size_t)W->n * 8));
  if (!walked && !W->prod32) TB_TRY(pr_alloc((void **)&W->prod32, (size_t)W->n * 4));
  PrMat<double, double> m;
  TB_TRY((solver_matrix<double, double>(A, static_cast<const double *>(A->values[0]), walked, W->prod, &m)));
  PrMat<V, float> mi;
  TB_TRY((solver_matrix<V, float>(A, static_cast<const V *>(A->values[store_index(store)]), walked, W->prod32, &mi)));
  TB_TRY(pr_partials(W, m.layout == kPrItems ? m.plan.n_chunked : mi.layout == kPrItems ? mi.plan.n_chunked : 0));
  a.x[0] = W->x[0];
  a.x[1] = W->x[1];
  a.mixed = 1;
  a.r32 = W->r;
  a.e32 = W->e[0];
  PrArgs<float> in;
  std::memset(&in, 0, sizeof in);
  in.x[0] = W->e[0];
  in.x[1] = W->e[1];
  for (int i = 0; i < 3; ++i) {
    in.g[i] = W->eg[i];
    in.r[i] = W->er[i];
  }
  in.dmask = W->dmask;
  in.rvec = W->r;
  in.x64 = W->x[0];
  in.limit = walked ? kInnerMax : 1;
  a.init = 1;
  a.limit = walked ? 1 : 0;
  if (!walked) {
    TB_TRY((launch_solver<kSweepDang, double, double, false>(A, m, a, W, W->stream)));
    a.init = 0;
    a.limit = 1;
  }
  for (int round = 0;; ++round) {
    if (!walked) TB_TRY(spmv_dispatch(A, TBSLA_F64, TBSLA_F64, W->x[0], TBSLA_F64, W->prod, 0, W->stream));
    TB_TRY((launch_solver<kSweepDang, double, double, false>(A, m, a, W, W->stream)));
    a.init = 0;
    // three corrections bring an FP32 store to 1e-12: the host looks after
    // the fourth FP64 sweep, then after each
    if (!walked || round >= 3) {
      TB_TRY(pr_wait(A, W));
      if (W->ctl_host->done) return TBSLA_OK;
    }
    if (walked) {
      TB_TRY((launch_solver<kSweepInner, V, float, AA>(A, mi, in, W, W->stream)));
      continue;
    }
    for (int k = 0;;) {
      for (int j = 0; j < check_every; ++j, ++k) {
        TB_TRY(spmv_dispatch(A, store, TBSLA_F32, AA ? W->e[0] : W->e[k & 1], TBSLA_F32, W->prod32, 0, W->stream));
        TB_TRY((launch_solver<kSweepInner, V, float, AA>(A, mi, in, W, W->stream)));
      }
      TB_TRY(pr_wait(A, W));
      if (W->ctl_host->inner_done) break;
    }
  }
}

tbsla_status_t pr_out_buffer(tbsla_matrix *A, double **out) {
  if (!A->pr_out) TB_TRY(dev_alloc(A, (void **)&A->pr_out, (size_t)A->n_col * sizeof(double)));
  *out = A->pr_out;
  return TBSLA_OK;
}

}  // namespace

tbsla_status_t pr_relabelled(tbsla_matrix *A, tbsla_matrix **B);

}  // namespace tbsla

using namespace tbsla;

// The solve on A itself; d_out[v] = the result at newid[v] (v when NULL).
static tbsla_status_t pagerank_impl(tbsla_matrix *A, const tbsla_pagerank_params_t *p, const int *nodes,
                                    int n_nodes, double *d_out, const int *newid, tbsla_pagerank_result_t *res,
                                    cudaStream_t user, const double *d_teleport) {
  PrWork *W = nullptr;
  TB_TRY(pr_setup(A, &W));
  TimingOff timing_off(A);
  TB_TRY(pr_order(W, user));
  const int n = W->n;
  const int K = p->check_every > 0 ? (p->check_every + 1) / 2 * 2 : 8;  // sweeps per look of the host, unwalked layouts
  PrArgs<double> a;
  std::memset(&a, 0, sizeof a);
  PrCtl &c = a.ctl0;
  c.beta = p->beta;
  c.tol = p->tol;
  c.inv_n = 1.0 / n;
  c.max_iter = p->max_iter;
  c.inner_max = kInnerMax;
  // the inner tolerance relative to ||r||: with accelerated inner solves an
  // FP32 store is solved further (each correction then gains about four
  // decades; R-MAT 2^20: 3 FP64 + 11 FP32 sweeps against 26 plain FP64
  // sweeps), a BF16 store as before (its model error bounds the gain)
  c.inner_eta = p->precision == TBSLA_BF16 ? 0.05 : p->accel ? 1e-4 : 0.01;
  c.tele_scale = (1.0 - p->beta) / (nodes ? n_nodes : n);
  c.done = p->max_iter == 0;
  a.dmask = W->dmask;
  a.out = d_out;
  a.newid = newid;
  a.tvec = d_teleport;
  if (nodes) {
    TB_CHECK(n_nodes > 0, "empty node list");
    std::vector<unsigned char> mask((size_t)n, 0);
    for (int k = 0; k < n_nodes; ++k)
      if (nodes[k] >= 0 && nodes[k] < n) mask[(size_t)nodes[k]] = 1;
    TB_CUDA(cudaMemcpyAsync(W->tmask, mask.data(), (size_t)n, cudaMemcpyHostToDevice, W->stream));
    TB_CUDA(cudaStreamSynchronize(W->stream));
    a.tmask = W->tmask;
  }
  if (p->precision != TBSLA_F64) {
    if (p->precision == TBSLA_F32 && p->accel) TB_TRY((run_mixed<float, true>(A, W, a, TBSLA_F32, K)));
    else if (p->precision == TBSLA_F32) TB_TRY((run_mixed<float, false>(A, W, a, TBSLA_F32, K)));
    else if (p->accel) TB_TRY((run_mixed<__nv_bfloat16, true>(A, W, a, TBSLA_BF16, K)));
    else TB_TRY((run_mixed<__nv_bfloat16, false>(A, W, a, TBSLA_BF16, K)));
  } else if (p->mode == TBSLA_PR_REFERENCE) {
    TB_TRY((run_f64<kSweepRef, false>(A, W, a, K)));
  } else if (p->mode == TBSLA_PR_TELEPORT) {
    if (p->accel) TB_TRY((run_f64<kSweepTele, true>(A, W, a, K)));
    else TB_TRY((run_f64<kSweepTele, false>(A, W, a, K)));
  } else {
    if (p->accel) TB_TRY((run_f64<kSweepDang, true>(A, W, a, K)));
    else TB_TRY((run_f64<kSweepDang, false>(A, W, a, K)));
  }
  if (res) {
    const PrCtl &h = *W->ctl_host;
    res->iterations = p->precision == TBSLA_F64 ? h.iter : h.f64_sweeps + h.inner_total;
    res->iterations_f64 = h.f64_sweeps;
    res->residual = h.resid;
    res->converged = h.converged;
  }
  return TBSLA_OK;
}

namespace tbsla {
tbsla_status_t ensure_transpose(tbsla_matrix *A, tbsla_matrix **T);
tbsla_status_t grad_values_f64(const tbsla_matrix *A, const double *a, const double *b, double scale, double *out,
                               cudaStream_t s);
}  // namespace tbsla

// The adjoint of the TBSLA_PR_TELEPORT fixed point (see tbsla_gb300.h).
static tbsla_status_t adjoint_impl(tbsla_matrix *A, const tbsla_pagerank_params_t *p, const double *d_v,
                                   const double *d_x, const double *d_w, double *d_gvals, double *d_gv,
                                   tbsla_pagerank_result_t *res, cudaStream_t user) {
  TB_CHECK(A && p && d_x && d_w, "NULL argument");
  TB_CHECK(A->format == TBSLA_FMT_CSR && A->csr_variant == 0, "the adjoint needs a CSR handle (default variant)");
  TB_CHECK(A->n_row == A->n_col && A->n_col > 0, "the adjoint needs a square matrix");
  TB_CHECK(A->values[0], "the adjoint needs the F64 value store");
  TB_CHECK(p->max_iter >= 0, "max_iter < 0");
  TB_CHECK(p->accel == 0 || p->accel == 1, "accel = %d not 0 or 1", p->accel);
  TB_CUDA(cudaSetDevice(A->device));
  PrWork *W = nullptr;
  TB_TRY(pr_setup(A, &W));
  tbsla_matrix *T = nullptr;
  TB_TRY(ensure_transpose(A, &T));
  TB_CHECK(T->stored > 0, "the adjoint needs a matrix with entries");
  const int n = W->n;
  if (!W->lam) TB_TRY(pr_alloc((void **)&W->lam, (size_t)n * 8));
  TB_TRY(pr_order(W, user));
  cudaStream_t s = W->stream;
  PrArgs<double> a;
  std::memset(&a, 0, sizeof a);
  PrCtl &c = a.ctl0;
  c.beta = p->beta;
  c.tol = p->tol;
  c.inv_n = 1.0 / n;
  c.max_iter = p->max_iter;
  c.done = p->max_iter == 0;
  a.dmask = W->dmask;
  a.tvec = d_v;
  a.w = d_w;
  a.out = W->lam;
  if (p->accel) TB_TRY((run_f64<kSweepAdj, true>(T, W, a, 8)));
  else TB_TRY((run_f64<kSweepAdj, false>(T, W, a, 8)));
  const PrCtl &h = *W->ctl_host;
  if (d_gv) {
    // dL/dv = (beta * d . x + 1 - beta) * lambda
    pr_mass_kernel<<<kMassBlocks, 256, 0, s>>>(d_x, n, W->dmask, W->partials);
    pr_scale_to_kernel<<<kMassBlocks, 256, 0, s>>>(W->lam, n, W->partials, kMassBlocks, p->beta, d_gv);
    TB_CUDA(cudaGetLastError());
  }
  if (d_gvals) TB_TRY(grad_values_f64(A, W->lam, d_x, p->beta, d_gvals, s));
  TB_CUDA(cudaStreamSynchronize(s));
  if (res) {
    res->iterations = h.iter;
    res->iterations_f64 = h.iter;
    res->residual = h.resid;
    res->converged = h.converged;
  }
  return TBSLA_OK;
}

// PageRank of A, on its relabelled copy when there is one (pr_relabel.cu);
// *result points to the vector in A's labels (d_out, or a buffer of A's).
// The reference mode never takes the copy: relabelling reorders every row's
// sum and the block sums of the max-normalised residual, and the reference's
// iteration count (Matrix.cpp:13-114) moves with that order near epsilon.
static tbsla_status_t pagerank_entry(tbsla_matrix *A, const tbsla_pagerank_params_t *p, const int *nodes,
                                     int n_nodes, double *d_out, tbsla_pagerank_result_t *res, cudaStream_t user,
                                     const double **result, const double *d_teleport = nullptr) {
  TB_CHECK(A && p, "NULL argument");
  TB_CHECK(A->n_row == A->n_col, "PageRank needs a square matrix (%d x %d)", A->n_row, A->n_col);
  TB_CHECK(A->n_col > 0, "empty matrix");
  TB_CHECK(p->max_iter >= 0, "max_iter < 0");
  TB_CHECK(p->mode == TBSLA_PR_REFERENCE || p->mode == TBSLA_PR_DANGLING || p->mode == TBSLA_PR_TELEPORT,
           "unknown PageRank mode %d", p->mode);
  TB_CHECK(p->mode != TBSLA_PR_TELEPORT || (d_teleport && p->precision == TBSLA_F64),
           "the teleport mode needs a teleport vector and FP64");
  TB_CHECK(p->precision == TBSLA_F64 || p->precision == TBSLA_F32 || p->precision == TBSLA_BF16, "bad precision");
  TB_CHECK(p->precision == TBSLA_F64 || p->mode == TBSLA_PR_DANGLING, "reduced precision needs TBSLA_PR_DANGLING");
  TB_CHECK(p->accel == 0 || (p->accel == 1 && p->mode != TBSLA_PR_REFERENCE && nodes == nullptr),
           "accel = %d: Anderson acceleration (1) is for the dangling and teleport modes", p->accel);
  TB_CHECK(A->values[0], "PageRank needs the F64 value store");
  TB_CHECK(p->precision == TBSLA_F64 || A->values[store_index((tbsla_dtype_t)p->precision)],
           "the requested reduced-precision value store is not present");
  TB_CHECK(nodes == nullptr || p->mode == TBSLA_PR_REFERENCE, "node lists are for the reference mode");
  TB_CUDA(cudaSetDevice(A->device));
  double *out = d_out;
  if (!out) TB_TRY(pr_out_buffer(A, &out));
  tbsla_matrix *B = nullptr;
  if (!d_teleport && p->mode != TBSLA_PR_REFERENCE) TB_TRY(pr_relabelled(A, &B));
  TB_TRY(pagerank_impl(B ? B : A, p, nodes, n_nodes, out, B ? A->pr_newid : nullptr, res, user, d_teleport));
  if (result) *result = out;
  return TBSLA_OK;
}

extern "C" {

tbsla_status_t tbsla_pagerank(const tbsla_matrix_t *A, const tbsla_pagerank_params_t *p, double *d_out,
                              tbsla_pagerank_result_t *result, void *stream) {
  return pagerank_entry(const_cast<tbsla_matrix *>(A), p, nullptr, 0, d_out, result, (cudaStream_t)stream,
                        nullptr);
}

tbsla_status_t tbsla_pagerank_teleport(const tbsla_matrix_t *A, const tbsla_pagerank_params_t *p,
                                       const double *d_v, double *d_out, tbsla_pagerank_result_t *result,
                                       void *stream) {
  TB_CHECK(p && d_v, "NULL argument");
  tbsla_pagerank_params_t q = *p;
  q.mode = TBSLA_PR_TELEPORT;
  q.precision = TBSLA_F64;
  return pagerank_entry(const_cast<tbsla_matrix *>(A), &q, nullptr, 0, d_out, result, (cudaStream_t)stream,
                        nullptr, d_v);
}

tbsla_status_t tbsla_pagerank_adjoint(const tbsla_matrix_t *A, const tbsla_pagerank_params_t *p,
                                      const double *d_v, const double *d_x, const double *d_w,
                                      double *d_grad_values, double *d_grad_v,
                                      tbsla_pagerank_result_t *result, void *stream) {
  return adjoint_impl(const_cast<tbsla_matrix *>(A), p, d_v, d_x, d_w, d_grad_values, d_grad_v, result,
                      (cudaStream_t)stream);
}

tbsla_status_t tbsla_pagerank_host(tbsla_matrix_t *A, const tbsla_pagerank_params_t *p, double *out,
                                   int64_t n_out, tbsla_pagerank_result_t *result) {
  TB_CHECK(A && out, "NULL argument");
  TB_CHECK(n_out >= A->n_col, "output has %lld entries, need %d", (long long)n_out, A->n_col);
  std::lock_guard<std::mutex> lk(A->host_mu);
  const double *r = nullptr;
  TB_TRY(pagerank_entry(A, p, nullptr, 0, nullptr, result, nullptr, &r));
  TB_CUDA(cudaMemcpy(out, r, (size_t)A->n_col * 8, cudaMemcpyDeviceToHost));
  return TBSLA_OK;
}

tbsla_status_t tbsla_personalized_pagerank_host(tbsla_matrix_t *A, const tbsla_pagerank_params_t *p,
                                                const int *nodes, int n_nodes, double *out, int64_t n_out,
                                                tbsla_pagerank_result_t *result) {
  TB_CHECK(A && out && nodes, "NULL argument");
  TB_CHECK(n_out >= A->n_col, "output has %lld entries, need %d", (long long)n_out, A->n_col);
  std::lock_guard<std::mutex> lk(A->host_mu);
  tbsla_pagerank_params_t q = *p;
  q.mode = TBSLA_PR_REFERENCE;
  q.precision = TBSLA_F64;
  const double *r = nullptr;
  TB_TRY(pagerank_entry(A, &q, nodes, n_nodes, nullptr, result, nullptr, &r));
  TB_CUDA(cudaMemcpy(out, r, (size_t)A->n_col * 8, cudaMemcpyDeviceToHost));
  return TBSLA_OK;
}

}  // extern "C"
