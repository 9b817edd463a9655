// csr_direct.cuh -- direct CSR SpMV kernels for sm_103a (the default CSR path).
//
// Rows are binned at creation by length:
//   short (<= kShortRow nonzeros), plain FP64 products of rows averaging at
//     least kPairMinRow entries: two lanes per row (csr_pair_kernel, below).
//   short, otherwise: one thread per row, walking its row in
//     chunks of eight entries with 16-byte loads straight from global memory.
//     Lanes of a warp hold neighbouring rows; the loads of one chunk are
//     issued together, so a sector's second use hits the line already in
//     flight in L1: L1 does the coalescing, no shared memory and no block
//     barrier are involved.  The row is summed in
//     its stored order with one FMA per nonzero (the order of
//     MatrixCSR::Ax, src/cpp/matrix/MatrixCSR.cpp:133-139).
//   long (<= kChunk): a group of L lanes per row, L = 4, 8, 32 or a block of
//     256 by length class (kGroupLimit, kManyLimit), lanes striding the row, partial sums
//     combined in a fixed order inside the group.
//   huge (> kChunk): the row is cut into chunks of kChunk nonzeros, a block
//     per chunk writing a partial; csr_chunk_fixup_kernel adds the partials of
//     each row in chunk order.
// Matrices with long rows run all of it in one launch (csr_mixed_kernel).
// The groups exist for the FP64 pipe (2 lane-operations per clock per SM on
// GB300; a warp instruction costs the same with 1 or 32 lanes active): one
// warp per row would spend ~10 FP64 warp instructions per row on its
// reduction and epilogue, more than the products of a 100-entry row.
// Row data is read through L1 with the default cache policy, the gathered x
// with a fractional evict-last L2 policy, y written with streaming stores.
// No atomics: results do not depend on scheduling.
#pragma once

#include <type_traits>

#include "spmv_kernels.cuh"

namespace tbsla {

constexpr int kShortRow = 32;
constexpr int kChunk = 8192;
// length classes of the long rows: class c takes rows of at most
// kGroupLimit[c] entries with kGroupLanes[c] lanes each (chunks: class 3)
constexpr int kGroupClasses = 4;
constexpr int kGroupLimit[kGroupClasses] = {96, 256, 1024, kChunk};
constexpr int kGroupLanes[kGroupClasses] = {4, 8, 32, 256};
// Rows of up to 1792 entries join the class of 32 lanes where there are as many as
// fill the GPU with warps: a block a row leaves much of its time to the sums of
// the lanes (rows of 1500 entries, 32 lanes / a block: 16384 of them 64 / 77 us in
// FP64, 46 / 51 in FP32, 45 / 56 in BF16; 30000 168 / 155, 78 / 89, 75 / 98; 8000 34 /
// 42 and 28 / 28; 4000 24 / 26 and 18 / 15).  Of 2000 entries 30000 rows take
// 224 us in FP64 by 32 lanes, 206 by blocks.
constexpr int kManyRows = 8192, kManyLimit = 1792;

__device__ __forceinline__ float bf16_lo(unsigned w) { return __bfloat162float(__ushort_as_bfloat16((unsigned short)(w & 0xffffu))); }
__device__ __forceinline__ float bf16_hi(unsigned w) { return __bfloat162float(__ushort_as_bfloat16((unsigned short)(w >> 16))); }

// eight entries from an 8-aligned index with 16-byte loads through L1 and the
// default cache policy (arrays carry 64 bytes of padding, so a group may run
// past the last entry).  A lane reads each sector in two pieces; L1/L2 keep
// the line between them.  Explicit L2 eviction hints were measured worse
// here: an evict-first hint lets L2 drop the line between the two reads
// (DRAM traffic x2.5), and 32-byte loads with an evict-normal policy ran 20%
// slower.  FP64 values and the column indices ask for 256-byte L2 prefetches:
// neutral at the default L2 fetch granularity, and they keep the streams
// wide when the process lowers it to 32 bytes for the gathers
// (tbsla_set_l2_fetch_granularity).
__device__ __forceinline__ void ld_vals8(const double *p, double (&v)[8]) {
  #pragma unroll
  for (int h = 0; h < 4; ++h)
    asm("ld.global.nc.L2::256B.v2.f64 {%0,%1}, [%2];" : "=d"(v[2 * h]), "=d"(v[2 * h + 1]) : "l"(p + 2 * h));
}
__device__ __forceinline__ void ld_vals8(const float *p, float (&v)[8]) {
  asm("ld.global.nc.L2::256B.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "l"(p));
  asm("ld.global.nc.L2::256B.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]) : "l"(p + 4));
}
__device__ __forceinline__ void ld_vals8(const __nv_bfloat16 *p, float (&v)[8]) {
  unsigned w[4];
  asm("ld.global.nc.L2::256B.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "l"(p));
  #pragma unroll
  for (int h = 0; h < 4; ++h) { v[2 * h] = bf16_lo(w[h]); v[2 * h + 1] = bf16_hi(w[h]); }
}
__device__ __forceinline__ void ld_cols8(const int *c, int (&col)[8]) {
  asm("ld.global.nc.L2::256B.v4.s32 {%0,%1,%2,%3}, [%4];" : "=r"(col[0]), "=r"(col[1]), "=r"(col[2]), "=r"(col[3]) : "l"(c));
  asm("ld.global.nc.L2::256B.v4.s32 {%0,%1,%2,%3}, [%4];" : "=r"(col[4]), "=r"(col[5]), "=r"(col[6]), "=r"(col[7]) : "l"(c + 4));
}
// two entries from an even index
__device__ __forceinline__ void ld_vals2(const double *p, double (&v)[2]) {
  const double2 d = __ldg(reinterpret_cast<const double2 *>(p));
  v[0] = d.x; v[1] = d.y;
}
__device__ __forceinline__ void ld_vals2(const float *p, float (&v)[2]) {
  const float2 d = __ldg(reinterpret_cast<const float2 *>(p));
  v[0] = d.x; v[1] = d.y;
}
__device__ __forceinline__ void ld_vals2(const __nv_bfloat16 *p, float (&v)[2]) {
  const unsigned w = __ldg(reinterpret_cast<const unsigned *>(p));
  v[0] = bf16_lo(w); v[1] = bf16_hi(w);
}

// One row, one thread.  Rows of eight or more entries go in groups of eight
// aligned to eight, all loads of a group issued together; shorter rows go in
// aligned pairs, which neighbouring lanes read as contiguous 16-byte pieces.
// Entries outside [a, b) of a group are masked (no gather, no FMA).  The row
// is summed in stored order, one FMA per entry.
template <int G, typename V, typename XT, typename Acc>
__device__ __forceinline__ Acc row_groups(const int *__restrict__ colidx, const V *__restrict__ values,
                                          const XT *__restrict__ x, int f_col, int a, int b, uint64_t keep) {
  using Ld = typename std::conditional<sizeof(V) == 8, double, float>::type;
  Acc acc = 0;
  for (int base = a & ~(G - 1); base < b; base += G) {
    Ld v[G];
    int col[G];
    if constexpr (G == 2) {
      ld_vals2(values + base, v);
      const int2 c = __ldg(reinterpret_cast<const int2 *>(colidx + base));
      col[0] = c.x; col[1] = c.y;
    } else {
      ld_vals8(values + base, v);
      ld_cols8(colidx + base, col);
    }
    Acc xv[G];
    #pragma unroll
    for (int e = 0; e < G; ++e) {
      const int k = base + e;
      xv[e] = (k >= a && k < b) ? to_acc(ld_keep(x + (col[e] - f_col), keep), Acc()) : Acc(0);
    }
    #pragma unroll
    for (int e = 0; e < G; ++e) {
      const int k = base + e;
      if (k >= a && k < b) acc = fma_acc((Acc)v[e], xv[e], acc);
    }
  }
  return acc;
}

template <typename V, typename XT, typename Acc>
__device__ __forceinline__ Acc row_sum_thread(const int *__restrict__ colidx, const V *__restrict__ values,
                                              const XT *__restrict__ x, int f_col, int a, int b,
                                              uint64_t keep) {
  if (b - a >= 8) return row_groups<8, V, XT, Acc>(colidx, values, x, f_col, a, b, keep);
  return row_groups<2, V, XT, Acc>(colidx, values, x, f_col, a, b, keep);
}

// every row short: one row per thread
template <typename V, typename XT, typename Epi>
__global__ void __launch_bounds__(256) csr_short_kernel(int n_rows,
                                                       const int *__restrict__ rowptr,
                                                       const int *__restrict__ colidx,
                                                       const V *__restrict__ values,
                                                       const XT *__restrict__ x, int f_col, XKeep x_keep,
                                                       Epi epi) {
  using Acc = typename Epi::Acc;
  const uint64_t keep = policy_keep(x_keep, x);
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n_rows; t += stride) {
    const int r = (int)t;
    const int a = __ldg(rowptr + r), b = __ldg(rowptr + r + 1);
    epi.emit(r, row_sum_thread<V, XT, Acc>(colidx, values, x, f_col, a, b, keep));
  }
}

// Short rows, two adjacent lanes per row: the row's aligned groups (of eight
// entries, or of two for rows under eight) are split in halves, each lane
// sums its half in stored order, and the row is first half + second half (a
// fixed order: results do not depend on scheduling, but round differently
// from the one-lane sum).  A warp's load instruction touches 16 rows' lines
// instead of 32, for one more FP64 add per row.
// the default uses the pairs for FP64 plain products when short rows
// average at least this many entries (cqmat c=16: 4889 vs 4378 GB/s with
// 32-byte L2 fetches; cdiag, 2 per row: 2516 vs 4647 -- a lane idles)
constexpr int kPairMinRow = 8;

template <typename V, typename XT, typename Acc>
__device__ __forceinline__ Acc row_half(const int *__restrict__ colidx, const V *__restrict__ values,
                                        const XT *__restrict__ x, int f_col, int a, int b, int half,
                                        uint64_t keep) {
  const int sh = b - a >= 8 ? 3 : 1;
  const int g0 = a >> sh, g1 = (b + (1 << sh) - 1) >> sh, gm = g0 + ((g1 - g0 + 1) >> 1);
  const int lo = half ? max(a, gm << sh) : a, hi = half ? b : min(b, gm << sh);
  if (lo >= hi) return Acc(0);
  if (sh == 3) return row_groups<8, V, XT, Acc>(colidx, values, x, f_col, lo, hi, keep);
  return row_groups<2, V, XT, Acc>(colidx, values, x, f_col, lo, hi, keep);
}

template <typename V, typename XT, typename Epi>
__global__ void __launch_bounds__(256) csr_pair_kernel(int n_rows,
                                                      const int *__restrict__ rowptr,
                                                      const int *__restrict__ colidx,
                                                      const V *__restrict__ values,
                                                      const XT *__restrict__ x, int f_col, XKeep x_keep,
                                                      Epi epi) {
  using Acc = typename Epi::Acc;
  const uint64_t keep = policy_keep(x_keep, x);
  const int half = threadIdx.x & 1;
  const unsigned pair = 3u << ((threadIdx.x & 31) & ~1);  // both lanes of a pair always run together
  const int64_t stride = ((int64_t)gridDim.x * blockDim.x) >> 1;
  for (int64_t t = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 1; t < n_rows; t += stride) {
    const int r = (int)t;
    const int a = __ldg(rowptr + r), b = __ldg(rowptr + r + 1);
    const Acc mine = row_half<V, XT, Acc>(colidx, values, x, f_col, a, b, half, keep);
    const Acc other = __shfl_xor_sync(pair, mine, 1);
    if (!half) epi.emit(r, mine + other);
  }
}

// Tiny rows: every row in order and at most T entries (T = 2 or 4).  A warp
// takes a tile of 32 R rows (R = 8 / T), lane l rows l, l + 32, ..., so
// each load instruction covers 32 consecutive rows; a lane has the bounds,
// entries and gathers of its R rows in flight together (one row per thread
// leaves three dependent loads per row in flight: cdiag rows of two entries
// stayed latency-bound at two thirds of the HBM rate).  Each row is summed
// in stored order, one FMA per entry: the one-thread-per-row arithmetic.
// (kTinyRow, the longest row it takes, is in common.cuh.)

template <int T, typename V, typename XT, typename Epi>
__global__ void __launch_bounds__(256) csr_tiny_kernel(int n_rows, const int *__restrict__ rowptr,
                                                      const int *__restrict__ colidx,
                                                      const V *__restrict__ values,
                                                      const XT *__restrict__ x, int f_col, XKeep x_keep,
                                                      Epi epi) {
  using Acc = typename Epi::Acc;
  constexpr int R = 8 / T;
  const int64_t base = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32 * (32 * R);
  if (base < n_rows) {
    const uint64_t keep = policy_keep(x_keep, x);
    const int r0 = (int)base + (threadIdx.x & 31);
    int a[R], b[R];
    #pragma unroll
    for (int q = 0; q < R; ++q) {
      const int r = r0 + 32 * q;
      a[q] = r < n_rows ? __ldg(rowptr + r) : 0;
      b[q] = r < n_rows ? __ldg(rowptr + r + 1) : 0;
    }
    V v[R][T];
    int c[R][T];
    #pragma unroll
    for (int q = 0; q < R; ++q) {
      #pragma unroll
      for (int t = 0; t < T; ++t) {
        const int k = a[q] + t;
        const bool in = k < b[q];
        c[q][t] = in ? ld_ell<false>(colidx + k) : f_col;  // read-only, 256-byte L2 prefetch
        v[q][t] = in ? ld_ell<false>(values + k) : V(0);
      }
    }
    Acc xv[R][T];
    #pragma unroll
    for (int q = 0; q < R; ++q) {
      #pragma unroll
      for (int t = 0; t < T; ++t)
        xv[q][t] = a[q] + t < b[q] ? to_acc(ld_keep(x + (c[q][t] - f_col), keep), Acc()) : Acc(0);
    }
    #pragma unroll
    for (int q = 0; q < R; ++q) {
      Acc acc = 0;
      #pragma unroll
      for (int t = 0; t < T; ++t)
        if (a[q] + t < b[q]) acc = fma_acc(to_acc(v[q][t], Acc()), xv[q][t], acc);
      if (r0 + 32 * q < n_rows) epi.emit(r0 + 32 * q, acc);
    }
  }
}

// The same share without the next step's loads in flight, for FP64 and FP32 groups
// of a whole warp where there are thousands (kPlainItems): the loads of the SM's other
// warps overlap with it, and the shorter loop wins (16384 rows of 900 entries: 44
// us against 49 in FP64, 31.5 / 34.2 in FP32).  With fewer of them, narrower
// groups and BF16 the loads ahead stay (R-MAT 2^16 FP64: 15.3 us, 17.8 without; 2^20
// banded rows of 48, FP32: 103, 121; 16384 rows of 900, BF16: 29.6, 31.5).
template <int L, typename V, typename XT, typename Acc>
__device__ __forceinline__ Acc range_sum_plain(const int *__restrict__ colidx, const V *__restrict__ values,
                                               const XT *__restrict__ x, int f_col, int a, int b, int lane,
                                               uint64_t keep) {
  Acc acc = 0;
  #pragma unroll 4
  for (int64_t k = (int64_t)a + lane; k < b; k += L)
    acc = fma_acc(to_acc(ld_stream(values + k), Acc()), to_acc(ld_keep(x + (ld_stream(colidx + k) - f_col), keep), Acc()), acc);
  return acc;
}

// A lane's share of entries [a, b) of a group of L lanes: entries a + lane,
// a + lane + L, ..., one FMA per entry in that order.  Four entries go
// together, their gathers in flight with the next four's columns and values.
template <int L, typename V, typename XT, typename Acc>
__device__ __forceinline__ Acc range_sum_lane(const int *__restrict__ colidx, const V *__restrict__ values,
                                              const XT *__restrict__ x, int f_col, int a, int b, int lane,
                                              uint64_t keep) {
  constexpr int U = 4;
  Acc acc = 0;
  int c[U];
  V v[U];
  auto load = [&](int64_t k) {
    #pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool in = k + u * L < b;
      c[u] = in ? ld_stream(colidx + k + u * L) : -1;
      v[u] = in ? ld_stream(values + k + u * L) : V(0);
    }
  };
  load((int64_t)a + lane);
  for (int64_t k = (int64_t)a + lane; k < b; k += L * U) {
    Acc xv[U];
    V vv[U];
    bool in[U];
    #pragma unroll
    for (int u = 0; u < U; ++u) {
      in[u] = c[u] >= 0;
      vv[u] = v[u];
      xv[u] = in[u] ? to_acc(ld_keep(x + (c[u] - f_col), keep), Acc()) : Acc(0);
    }
    load(k + L * U);
    #pragma unroll
    for (int u = 0; u < U; ++u)
      if (in[u]) acc = fma_acc(to_acc(vv[u], Acc()), xv[u], acc);
  }
  return acc;
}

// One long row (or chunk) by a group of L lanes of a warp, items [first,
// first + n) dealt 256 / L to a block: items[i] = (row, begin, end, partial
// slot or -1).  A warp holds 32/L groups, so its FP64 reduction steps and the
// epilogue serve 32/L rows at once.
template <int L, bool kPlain, typename V, typename XT, typename Epi>
__device__ __forceinline__ void mixed_group(const int4 *__restrict__ items, int n, int block,
                                            const int *__restrict__ colidx, const V *__restrict__ values,
                                            const XT *__restrict__ x, int f_col, uint64_t keep, const Epi &epi) {
  using Acc = typename Epi::Acc;
  const int i = block * (256 / L) + (int)threadIdx.x / L, lane = threadIdx.x & (L - 1);
  const int4 it = i < n ? __ldg(items + i) : make_int4(-1, 0, 0, -1);
  Acc s = kPlain ? range_sum_plain<L, V, XT, Acc>(colidx, values, x, f_col, it.y, it.z, lane, keep)
                 : range_sum_lane<L, V, XT, Acc>(colidx, values, x, f_col, it.y, it.z, lane, keep);
  #pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, L);
  if (lane == 0 && it.x >= 0) epi.emit(it.x, s);
}

// Matrices with long rows, one launch: the blocks take, in this order, the
// block-wide items (a row above 1024 entries or a chunk each), the items of
// 32, 8 and 4 lanes, and the short rows (one lane each, or two: kPair), so
// that the longest items start first and the small classes fill the GPU
// together.  One launch per class left the classes one after the other
// and walked chunks of 8192 entries with 32 lanes: a ragged FP32 matrix of
// 600011 rows (8 million entries, 30 hub rows) took 150 us, 67 of them the 30
// hub rows.
struct MixedPlan {
  const int4 *items;
  int start[kGroupClasses + 1];  // items of class c: [start[c], start[c + 1])
  int first[kGroupClasses + 1];  // first block of class c (3, 2, 1, 0), [kGroupClasses]: of the short rows
  const int *rows;               // short rows
  int n_short;
};

constexpr int kPlainItems = 152 * 32;  // 32-lane items: a warp for half of the SMs' places

template <bool kPair, bool kPlain, typename V, typename XT, typename Epi>
__global__ void __launch_bounds__(256) csr_mixed_kernel(const MixedPlan p, const int *__restrict__ rowptr,
                                                       const int *__restrict__ colidx, const V *__restrict__ values,
                                                       const XT *__restrict__ x, int f_col, XKeep x_keep,
                                                       typename Epi::Acc *__restrict__ partials, Epi epi) {
  using Acc = typename Epi::Acc;
  __shared__ Acc part[256];
  const uint64_t keep = policy_keep(x_keep, x);
  const int b = blockIdx.x;
  if (b < p.first[2]) {
    const int4 it = __ldg(p.items + p.start[3] + b);
    // FP64 without the loads ahead (16384 rows of 5000 entries: 173 us, 188 with; FP32 130, 120)
    if constexpr (sizeof(V) == 8)
      part[threadIdx.x] = range_sum_plain<256, V, XT, Acc>(colidx, values, x, f_col, it.y, it.z, threadIdx.x, keep);
    else
      part[threadIdx.x] = range_sum_lane<256, V, XT, Acc>(colidx, values, x, f_col, it.y, it.z, threadIdx.x, keep);
    __syncthreads();
    if (threadIdx.x < 32) {
      Acc s = part[threadIdx.x];
      #pragma unroll
      for (int u = 1; u < 8; ++u) s += part[threadIdx.x + 32 * u];
      #pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
      if (threadIdx.x == 0) {
        if (it.w < 0) epi.emit(it.x, s);
        else partials[it.w] = s;
      }
    }
  } else if (b < p.first[1]) {
    mixed_group<32, kPlain, V, XT, Epi>(p.items + p.start[2], p.start[3] - p.start[2], b - p.first[2], colidx, values, x, f_col, keep, epi);
  } else if (b < p.first[0]) {
    mixed_group<8, false, V, XT, Epi>(p.items + p.start[1], p.start[2] - p.start[1], b - p.first[1], colidx, values, x, f_col, keep, epi);
  } else if (b < p.first[4]) {
    mixed_group<4, false, V, XT, Epi>(p.items + p.start[0], p.start[1] - p.start[0], b - p.first[0], colidx, values, x, f_col, keep, epi);
  } else if constexpr (kPair) {
    const int64_t t = ((int64_t)(b - p.first[4]) * 256 + threadIdx.x) >> 1;
    const int half = threadIdx.x & 1;
    const unsigned pair = 3u << ((threadIdx.x & 31) & ~1);  // both lanes of a pair always run together
    if (t < p.n_short) {
      const int r = __ldg(p.rows + t);
      const int a = __ldg(rowptr + r), e = __ldg(rowptr + r + 1);
      const Acc mine = row_half<V, XT, Acc>(colidx, values, x, f_col, a, e, half, keep);
      const Acc other = __shfl_xor_sync(pair, mine, 1);
      if (!half) epi.emit(r, mine + other);
    }
  } else {
    const int64_t t = (int64_t)(b - p.first[4]) * 256 + threadIdx.x;
    if (t < p.n_short) {
      const int r = __ldg(p.rows + t);
      const int a = __ldg(rowptr + r), e = __ldg(rowptr + r + 1);
      epi.emit(r, row_sum_thread<V, XT, Acc>(colidx, values, x, f_col, a, e, keep));
    }
  }
}

// ---------------------------------------------------------------- staged
// Matrices whose rows are all short (<= kShortRow entries).  A warp takes
// tiles of 32 consecutive rows; a tile's entries are contiguous, and the warp
// copies them into its slice of shared memory with lane-per-entry copies
// (each line of row data read by one instruction, evict-first in L2 so that
// the streamed matrix leaves L2 to x).  Then each lane sums its own row from
// shared memory in stored order, one FMA per entry (the direct kernel's
// arithmetic: results are bit-identical), gathering x with the kept-fraction
// policy.  Slots are XOR-swizzled within groups of 16 entries, so lanes
// reading rows of 16 entries hit distinct banks.  Warps work independently;
// the block meets only in the epilogue's reduction.  (Per-element cp.async
// copies into two buffers per warp, overlapping the next tile's copies with
// the current sum, measured 1.5x slower than these register copies.)
constexpr int kStageWarps = 8;
constexpr int kStageBatch = 8;                // loads in flight per lane
constexpr int kStageCapMax = 32 * kShortRow;  // a tile's entries when every row is short

template <typename T> __device__ __forceinline__ T ld_first(const T *p, uint64_t pol);
template <> __device__ __forceinline__ double ld_first<double>(const double *p, uint64_t pol) {
  double v;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.L2::256B.f64 %0, [%1], %2;" : "=d"(v) : "l"(p), "l"(pol));
  return v;
}
template <> __device__ __forceinline__ float ld_first<float>(const float *p, uint64_t pol) {
  float v;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.L2::256B.f32 %0, [%1], %2;" : "=f"(v) : "l"(p), "l"(pol));
  return v;
}
template <> __device__ __forceinline__ int ld_first<int>(const int *p, uint64_t pol) {
  int v;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.L2::256B.s32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(pol));
  return v;
}
template <> __device__ __forceinline__ __nv_bfloat16 ld_first<__nv_bfloat16>(const __nv_bfloat16 *p, uint64_t pol) {
  unsigned short v;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.L2::256B.u16 %0, [%1], %2;" : "=h"(v) : "l"(p), "l"(pol));
  return __ushort_as_bfloat16(v);
}

__device__ __forceinline__ int stage_swz(int k) { return k ^ ((k >> 4) & 15); }

// dynamic shared memory of csr_stage_kernel for value type V and `cap` slots
template <typename V> constexpr size_t csr_stage_smem(int cap) {
  return (size_t)kStageWarps * cap * (sizeof(V) + sizeof(int));
}

// lane bounds of tile t: row r0+lane spans [lo, hi); lanes past the matrix
// (or a tile past the end) see empty rows
__device__ __forceinline__ void stage_bounds(const int *__restrict__ rowptr, int rows, int n_tiles, int t, int lane,
                                             int &lo, int &hi) {
  lo = hi = 0;
  if (t < n_tiles) {
    const int r0 = t << 5, nr = min(32, rows - r0);
    lo = __ldg(rowptr + r0 + min(lane, nr));
    hi = __ldg(rowptr + r0 + min(lane + 1, nr));
  }
}

template <typename V, typename XT, typename Acc>
__device__ __forceinline__ Acc stage_row_sum(const V *sv, const int *sc, int a, int b, const XT *__restrict__ x,
                                             int f_col, uint64_t keep) {
  Acc acc = 0;
  #pragma unroll 8
  for (int k = a; k < b; ++k) {
    const int sk = stage_swz(k);
    acc = fma_acc(to_acc(sv[sk], Acc()), to_acc(ld_keep(x + (sc[sk] - f_col), keep), Acc()), acc);
  }
  return acc;
}

template <typename V, typename XT, typename Epi>
__global__ void __launch_bounds__(kStageWarps * 32) csr_stage_kernel(int rows, const int *__restrict__ rowptr,
                                                                    const int *__restrict__ colidx,
                                                                    const V *__restrict__ values,
                                                                    const XT *__restrict__ x, int f_col,
                                                                    XKeep x_keep, int cap, Epi epi) {
  using Acc = typename Epi::Acc;
  extern __shared__ __align__(16) unsigned char stage_smem[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  V *sv = reinterpret_cast<V *>(stage_smem) + (size_t)wib * cap;
  int *sc = reinterpret_cast<int *>(stage_smem + (size_t)kStageWarps * cap * sizeof(V)) + (size_t)wib * cap;
  const uint64_t keep = policy_keep(x_keep, x), first = policy_evict_first();
  const int n_tiles = (rows + 31) >> 5;
  const int nw = gridDim.x * kStageWarps;
  int t = blockIdx.x * kStageWarps + wib;
  for (; t < n_tiles; t += nw) {
    int lo, hi;
    stage_bounds(rowptr, rows, n_tiles, t, lane, lo, hi);
    const int e0 = __shfl_sync(0xffffffffu, lo, 0), e1 = __shfl_sync(0xffffffffu, hi, 31);
    const int n = e1 - e0;  // <= cap by construction
    for (int k0 = 0; k0 < n; k0 += 32 * kStageBatch) {
      V v[kStageBatch];
      int c[kStageBatch];
      #pragma unroll
      for (int u = 0; u < kStageBatch; ++u) {
        const int k = k0 + u * 32 + lane;
        if (k < n) {
          v[u] = ld_first(values + e0 + k, first);
          c[u] = ld_first(colidx + e0 + k, first);
        }
      }
      #pragma unroll
      for (int u = 0; u < kStageBatch; ++u) {
        const int k = k0 + u * 32 + lane;
        if (k < n) {
          sv[stage_swz(k)] = v[u];
          sc[stage_swz(k)] = c[u];
        }
      }
    }
    __syncwarp();
    const Acc acc = stage_row_sum<V, XT, Acc>(sv, sc, lo - e0, hi - e0, x, f_col, keep);
    if ((t << 5) + lane < rows) epi.emit((t << 5) + lane, acc);
    __syncwarp();  // the next tile's copies overwrite the slots
  }
}

// y[row] = sum of the row's chunk partials in chunk order;
// huge[h] = (row, first slot), huge[n_huge].y = total slots
template <typename Epi>
__global__ void csr_chunk_fixup_kernel(const int2 *__restrict__ huge, int n_huge,
                                       const typename Epi::Acc *__restrict__ partials, Epi epi) {
  using Acc = typename Epi::Acc;
  const int h = blockIdx.x * blockDim.x + threadIdx.x;
  if (h < n_huge) {
    const int row = huge[h].x, first = huge[h].y, last = huge[h + 1].y;
    Acc s = partials[first];
    for (int c = first + 1; c < last; ++c) s += partials[c];
    epi.emit(row, s);
  }
}


// ------------------------------------------------------- sliced copy
// Every row short, few padded slots: a copy of the entries in ELL layout,
// slot j of every row stored together (rows padded to a multiple of 128,
// width = the longest row; padded slots hold column -1).  One warp per 32 R
// rows, lane l taking rows l, l + 32, ...: each slot's indices and values
// are R fully used 32-entry runs, and the gathers of neighbouring rows' band
// entries fall on neighbouring addresses.  Padded slots are skipped.  R = 2
// by default (two independent loads per slot and thread).  Each row is summed in its stored order, one FMA per entry (the
// order of MatrixCSR::Ax, src/cpp/matrix/MatrixCSR.cpp:133-139).
constexpr int kSellRows = 128;

template <int R, typename V, typename XT, typename Epi>
__global__ void __launch_bounds__(256) csr_sell_kernel(const int *__restrict__ cols, const V *__restrict__ vals,
                                                      int64_t stride, int width, const XT *__restrict__ x,
                                                      int f_col, int rows, XKeep x_keep, Epi epi) {
  using Acc = typename Epi::Acc;
  const int64_t base = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32 * (32 * R);
  const int lane = threadIdx.x & 31;
  if (base < rows) {
    const uint64_t keep = policy_keep(x_keep, x);
    const int r0 = (int)base + lane;
    Acc a[R];
    #pragma unroll
    for (int q = 0; q < R; ++q) a[q] = 0;
    #pragma unroll 4
    for (int j = 0; j < width; ++j) {
      const size_t off = (size_t)j * stride + r0;
      int c[R];
      V v[R];
      #pragma unroll
      for (int q = 0; q < R; ++q) {
        c[q] = ld_ell<false>(cols + off + 32 * q);
        v[q] = ld_ell<false>(vals + off + 32 * q);
      }
      #pragma unroll
      for (int q = 0; q < R; ++q)
        if (c[q] >= 0) a[q] = fma_acc(to_acc(v[q], Acc()), to_acc(ld_keep(x + (c[q] - f_col), keep), Acc()), a[q]);
    }
    #pragma unroll
    for (int q = 0; q < R; ++q)
      if (r0 + 32 * q < rows) epi.emit(r0 + 32 * q, a[q]);
  }
}

// the sliced copy of one array: entry rowptr[r] + j to slot j * stride + r
// (one thread per row)
template <typename T>
__global__ void sell_scatter_kernel(const int *__restrict__ rowptr, int64_t stride, int rows,
                                    const T *__restrict__ src, T *__restrict__ dst) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += (int64_t)gridDim.x * blockDim.x) {
    const int a = rowptr[r], b = rowptr[r + 1];
    for (int j = 0; j < b - a; ++j) dst[(size_t)j * stride + r] = src[a + j];
  }
}

}  // namespace tbsla
