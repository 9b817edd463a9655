// ppr_batch.cu -- many personalized PageRank vectors of one graph solved
// together (TBSLA_PR_TELEPORT form, one teleport set per vector).
//
// The k iterates are kept in tiles of KT columns (KT = 2, 4, 8, 16 or 32), each
// tile row-major: tile t, row i holds X[i*KT + c] for its KT vectors, so the
// gather of a column index brings all KT values in one contiguous segment.
// A group of G lanes sums a row, each lane VW consecutive vectors (16 bytes
// of the tile row): no cross-lane reduction, every lane does useful
// multiply-adds, and a warp sweeps 32 / G rows at once.  Rows longer than a
// chunk (PprPlan) are cut into chunks (partials + a fixup kernel) so that
// hub rows of power-law graphs spread over many groups.  The FP64 sweeps are
// bound by the FP64 pipe (2 operations per clock per SM: 64 vectors of R-MAT 2^17
// keep it 87 % busy, DRAM 12 %), the FP32 ones by the latency of their gathers
// (FP64 pipe 57 %: the dangling mass; L1 46 %).
//
// Anderson acceleration (p->accel = 1), per vector as in the one-vector
// solve: the sweep writes its output g and residual r = g - x into rings of
// three slots and sums r's dots with the two previous residuals; the
// finalize solves each vector's 3x3 normal equations (aa_coefficients) and
// the next input is the combination of the last three outputs.
//
// Per vector c with seed set P_c (v_c = 1/|P_c| on P_c):
//   x_c <- beta A x_c + (beta d.x_c + 1 - beta) v_c,
// stopped on its own when ||x_c - x_c,prev||_1 < tol (or max_iter sweeps);
// a stopped vector is frozen (its lanes copy the old value), and a tile
// whose vectors have all stopped skips its kernels.  Every check_every
// sweeps the host writes out the vectors that stopped and, when the ones
// still running fit in fewer tiles, repacks them (iterates, seeds, control
// state) so that no tile sweeps for one slow vector while its other lanes
// idle.  A column's arithmetic and its reduction order do not depend on its
// tile or lane, so repacking leaves every result bit for bit as it was.
// All sums have a fixed order: results do not depend on scheduling.
//
// Large skewed graphs run on the degree-relabelled copy (pr_relabel.cu);
// seeds are mapped in and the results gathered back to the original labels.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

#include "anderson.cuh"
#include "column_mask.cuh"
#include "product.cuh"

namespace tbsla {

tbsla_status_t pr_relabelled(tbsla_matrix *A, tbsla_matrix **B);

namespace {

constexpr int kPprChunkMin = 64, kPprChunkMax = 512;

struct ColCtl {
  double add;    // beta * d.x + cst of the current iterate
  double resid;  // last L1 change
  double tol;    // the column's stopping threshold
  int iter, done;
};
struct TileCtl {
  int done, iter;  // iter: sweeps run on the tile (parity of the buffer holding it)
  int ran;         // the last sweep ran on the tile (it was not stopped before)
  int pad;
};
// Anderson state of a column (accelerated solves): the next-sweep terms of
// the last three outputs and their residuals' Gram matrix, newest first; the
// weights of the next input in those outputs; residuals stored so far (0-3)
struct ColAa {
  double add[3];
  double gram[3][3];
  double coef[3];
  int hist, m;
};

// Lanes of the sweep kernels: each lane carries VW consecutive vectors (16
// bytes of a tile row, or the whole row when it is narrower), so a row takes
// G = KT / VW lanes and a warp sweeps 32 / G rows at once.
template <typename T, int KT>
struct PprLanes {
  static constexpr int VW = KT * (int)sizeof(T) >= 16 ? 16 / (int)sizeof(T) : KT;
  static constexpr int G = KT / VW;
};
template <typename T, int VW> struct PprVec;
template <> struct PprVec<double, 2> { using type = double2; };
template <> struct PprVec<float, 2> { using type = float2; };
template <> struct PprVec<float, 4> { using type = float4; };

template <typename T, int VW>
__device__ __forceinline__ void ppr_ld(const T *p, T (&v)[VW]) {
  using V = typename PprVec<T, VW>::type;
  const V q = __ldg(reinterpret_cast<const V *>(p));
  const T *s = reinterpret_cast<const T *>(&q);
  #pragma unroll
  for (int i = 0; i < VW; ++i) v[i] = s[i];
}
template <typename T, int VW>
__device__ __forceinline__ void ppr_st(T *p, const T (&v)[VW]) {
  using V = typename PprVec<T, VW>::type;
  V q;
  T *d = reinterpret_cast<T *>(&q);
  #pragma unroll
  for (int i = 0; i < VW; ++i) d[i] = v[i];
  *reinterpret_cast<V *>(p) = q;
}

// Per-column sums of a block into partials[(part*KT + c)*NV + v], for the NV
// values (resid, dangling mass, and with acceleration the residual dots
// r.r, r.r_prev, r.r_prev2) that each lane holds for its VW columns (lane l
// of a row group: columns l*VW .. l*VW+VW-1).  The warp's row groups are
// summed by shuffles, then the warps in order.
template <int KT, int VW, int NV>
__device__ __forceinline__ void block_columns(double (&v)[NV][VW], double *partials, int part) {
  constexpr int G = KT / VW;
  __shared__ double sh[8][32][NV];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  #pragma unroll
  for (int o = 16; o >= G; o >>= 1) {
    #pragma unroll
    for (int j = 0; j < NV; ++j)
      #pragma unroll
      for (int q = 0; q < VW; ++q) v[j][q] += __shfl_down_sync(0xffffffffu, v[j][q], o);
  }
  if (lane < G) {
    #pragma unroll
    for (int j = 0; j < NV; ++j)
      #pragma unroll
      for (int q = 0; q < VW; ++q) sh[warp][lane * VW + q][j] = v[j][q];
  }
  __syncthreads();
  if (threadIdx.x < KT) {
    double a[NV];
    #pragma unroll
    for (int j = 0; j < NV; ++j) a[j] = 0;
    const int nw = blockDim.x >> 5;
    for (int w = 0; w < nw; ++w)
      #pragma unroll
      for (int j = 0; j < NV; ++j) a[j] += sh[w][threadIdx.x][j];
    #pragma unroll
    for (int j = 0; j < NV; ++j) partials[((size_t)part * KT + threadIdx.x) * NV + j] = a[j];
  }
}

// the residual ring of an accelerated sweep: r0 receives r = y - x, r1 / r2
// hold the previous two sweeps' residuals
template <typename T>
struct PprRing {
  T *r0;
  const T *r1, *r2;
};

// A sweep's per-column constants for one lane's VW columns
template <int VW>
struct PprCols {
  double tele[VW];  // teleport term added at seed rows
  float tele_f[VW];  // the same rounded to FP32 (FP32 tiles)
  bool stopped[VW];
  int hist[VW];  // accelerated: residuals stored before this sweep
};
template <int VW, bool AA>
__device__ __forceinline__ void ppr_cols(PprCols<VW> &pc, int c, const ColCtl *col, const double *inv_size,
                                         const ColAa *aa) {
  #pragma unroll
  for (int q = 0; q < VW; ++q) {
    const ColCtl cc = col[c + q];
    pc.stopped[q] = cc.done != 0;
    pc.tele[q] = cc.add * inv_size[c + q];
    pc.tele_f[q] = (float)pc.tele[q];
    pc.hist[q] = AA ? aa[c + q].hist : 0;
  }
}

// The loads of a row's epilogue
template <typename T, int VW, bool AA>
struct PprRowIn {
  T old[VW], rh[VW], r1[VW], r2[VW];
  unsigned sd;
  bool dm;
};
template <typename T, int VW, bool AA>
__device__ __forceinline__ void ppr_row_in(PprRowIn<T, VW, AA> &in, int row, int KT, int c, const PprCols<VW> &pc,
                                           const T *xo, const unsigned *seeds, const unsigned char *dmask,
                                           const T *rhs, const PprRing<T> &ring) {
  const size_t at = (size_t)row * KT + c;
  ppr_ld<T, VW>(xo + at, in.old);
  if (rhs) ppr_ld<T, VW>(rhs + at, in.rh);
  in.sd = __ldg(seeds + row) >> c;
  in.dm = __ldg(dmask + row) != 0;
  if constexpr (AA) {
    int h = 0;
    #pragma unroll
    for (int q = 0; q < VW; ++q) h = max(h, pc.hist[q]);
    if (h >= 1) ppr_ld<T, VW>(ring.r1 + at, in.r1);
    if (h >= 2) ppr_ld<T, VW>(ring.r2 + at, in.r2);
  }
}

// New values of one finished row for a lane's VW columns:
//   y = beta acc + [seed row] tele + rhs (a stopped column keeps its value),
// their L1 change (res) and dangling mass (dm, FP64: it sets the next
// sweep's teleport term, so the fixed point); accelerated: r = y - x into
// the ring and its dots with the previous residuals, summed per thread in
// shared memory (dots[(j*VW + q)*256 + thread]: registers are the sweep's
// limit).  FP32 tiles compute y, the L1 change and the dots in FP32 (the
// per-thread sums cover a few hundred rows; the block and grid sums are
// FP64): the FP64 pipe, two operations per clock per SM, is kept for the
// dangling mass.
template <typename T, int VW, bool AA>
__device__ __forceinline__ void ppr_emit(int row, int KT, int c, const T (&acc)[VW], const PprCols<VW> &pc,
                                         const PprRowIn<T, VW, AA> &in, T *xn, double beta, bool has_rhs,
                                         const PprRing<T> &ring, T (&res)[VW], double (&dm)[VW], T *dots) {
  const size_t at = (size_t)row * KT + c;
  T y[VW];
  #pragma unroll
  for (int q = 0; q < VW; ++q) {
    if (pc.stopped[q]) {
      y[q] = in.old[q];
    } else {
      if constexpr (std::is_same<T, float>::value) {
        float t = ((in.sd >> q) & 1u) ? pc.tele_f[q] : 0.f;
        if (has_rhs) t += in.rh[q];
        y[q] = fmaf((float)beta, acc[q], t);
        res[q] += fabsf(y[q] - in.old[q]);
      } else {
        double t = ((in.sd >> q) & 1u) ? pc.tele[q] : 0.0;
        if (has_rhs) t += (double)in.rh[q];
        y[q] = (T)((double)beta * (double)acc[q] + t);
        res[q] += fabs((double)y[q] - (double)in.old[q]);
      }
    }
    if (in.dm) dm[q] += (double)y[q];
  }
  ppr_st<T, VW>(xn + at, y);
  if constexpr (AA) {
    T r[VW];
    #pragma unroll
    for (int q = 0; q < VW; ++q) r[q] = y[q] - in.old[q];
    ppr_st<T, VW>(ring.r0 + at, r);
    #pragma unroll
    for (int q = 0; q < VW; ++q) {
      T *dq = dots + (size_t)q * 256 + threadIdx.x;
      dq[0] += r[q] * r[q];
      if (pc.hist[q] >= 1) dq[VW * 256] += r[q] * in.r1[q];
      if (pc.hist[q] >= 2) dq[2 * VW * 256] += r[q] * in.r2[q];
    }
  }
}

// the per-thread sums of a sweep kernel in the layout of block_columns
template <typename T, int VW, int NV, bool AA>
__device__ __forceinline__ void ppr_gather_parts(const T (&res)[VW], const double (&dm)[VW], const T *dots,
                                                 double (&part)[NV][VW]) {
  #pragma unroll
  for (int q = 0; q < VW; ++q) {
    part[0][q] = (double)res[q];
    part[1][q] = dm[q];
  }
  if constexpr (AA)
    #pragma unroll
    for (int j = 0; j < 3; ++j)
      #pragma unroll
      for (int q = 0; q < VW; ++q) part[2 + j][q] = (double)dots[(j * VW + q) * 256 + threadIdx.x];
}

// What the kernels of one sweep need, tile t = blockIdx.y of the layout: every
// array holds the tiles one after another.  All tiles go in one launch, so
// that they fill the GPU together and a sweep costs as many launches as one
// tile's.
template <typename T>
struct PprSweep {
  const T *xo;               // iterates
  T *xn;                     // outputs
  PprRing<T> ring;
  const T *rhs;              // added to every sweep, or NULL
  const unsigned *seeds;
  const unsigned char *dmask;
  const ColCtl *col;
  const ColAa *aa;
  const double *inv_size;
  T *chunks;                 // sums of the rows' chunks
  double *partials;
  const TileCtl *tile;
  double beta;
  int n, slots, nparts;      // rows, chunk slots and partial slots of a tile
};

// Resident blocks per SM the sweep kernel is compiled for (its register
// budget, 64 registers): the sweeps are bound by the latency of their
// gathers, and resident warps keep them in flight (R-MAT 2^22, 256 vectors,
// FP64: 1 block per SM (144 registers) 1.77x the time of 4; 5 no faster)
template <typename T, bool AA>
constexpr int ppr_min_blocks() {
  return 4;
}

// items: (row, begin, end, chunk slot or -1).  A row group of G lanes takes
// an item, lane l its vectors l*VW .. l*VW+VW-1 (one 16-byte gather of the
// tile row per entry); each vector's sum is one FMA per entry in stored order.
// Items come in decreasing length (a tile row is whole lines, so their order
// costs no coalescing): the groups of a warp walk rows of one length and the
// longest start first.  Groups of eight lanes or more read eight entries with
// one load per array, a lane each, and share them by shuffles; narrower ones
// read four, every lane all of them.  Either way the step's gathers are all
// issued before its first multiply-add, the next item ahead.
template <typename T, int KT, bool AA>
__global__ void __launch_bounds__(256, ppr_min_blocks<T, AA>()) ppr_spmm_kernel(const int4 *__restrict__ items, int n_items,
                                                      const int *__restrict__ colidx, const T *__restrict__ values,
                                                      const PprSweep<T> p) {
  const int tl = blockIdx.y;
  if (*(volatile const int *)&p.tile[tl].done) return;
  constexpr int VW = PprLanes<T, KT>::VW, G = PprLanes<T, KT>::G, NV = AA ? 5 : 2;
  const int c = (threadIdx.x & (G - 1)) * VW;  // first vector of this lane
  const size_t off = (size_t)tl * p.n * KT;
  const T *__restrict__ xo = p.xo + off;
  T *__restrict__ xn = p.xn + off;
  const T *rhs = p.rhs ? p.rhs + off : nullptr;
  const PprRing<T> ring{AA ? p.ring.r0 + off : nullptr, AA ? p.ring.r1 + off : nullptr,
                        AA ? p.ring.r2 + off : nullptr};
  const unsigned *seeds = p.seeds + (size_t)tl * p.n;
  PprCols<VW> pc;
  ppr_cols<VW, AA>(pc, c, p.col + tl * KT, p.inv_size + tl * KT, p.aa + tl * KT);
  const int64_t ng = ((int64_t)gridDim.x * blockDim.x) / G;
  T res[VW];
  double dm[VW];
  #pragma unroll
  for (int q = 0; q < VW; ++q) {
    res[q] = 0;
    dm[q] = 0;
  }
  __shared__ T dots[AA ? 3 * VW * 256 : 1];
  if (AA)
    for (int j = 0; j < 3 * VW; ++j) dots[j * 256 + threadIdx.x] = 0;
  int64_t g = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / G;
  int4 it = g < n_items ? __ldg(items + g) : make_int4(0, 0, 0, -1);
  for (; g < n_items; g += ng) {
    const int4 nx = g + ng < n_items ? __ldg(items + g + ng) : make_int4(0, 0, 0, -1);
    T acc[VW];
    #pragma unroll
    for (int q = 0; q < VW; ++q) acc[q] = 0;
    if constexpr (G >= 8) {
      const unsigned mask = G == 32 ? 0xffffffffu : ((1u << (G & 31)) - 1u) << ((threadIdx.x & 31) & ~(G - 1));
      const int sl = threadIdx.x & (G - 1) & 7;
      for (int e = it.y; e < it.z; e += 8) {
        const int rem = it.z - e;
        const int cm = sl < rem ? __ldg(colidx + e + sl) : 0;
        const T vm = sl < rem ? __ldg(values + e + sl) : T(0);
        constexpr int H = 4;  // gathers in flight (registers)
        #pragma unroll
        for (int h = 0; h < 8; h += H) {
          T xj[H][VW];
          #pragma unroll
          for (int u = 0; u < H; ++u) {
            const int cj = __shfl_sync(mask, cm, h + u, G);
            if (h + u < rem) ppr_ld<T, VW>(xo + (size_t)cj * KT + c, xj[u]);
          }
          #pragma unroll
          for (int u = 0; u < H; ++u) {
            const T vj = __shfl_sync(mask, vm, h + u, G);
            if (h + u < rem)
              #pragma unroll
              for (int q = 0; q < VW; ++q) acc[q] = fma(vj, xj[u][q], acc[q]);
          }
        }
      }
    } else {
      for (int e = it.y; e < it.z; e += 4) {
        const int rem = it.z - e;
        int cj[4];
        T vj[4], xj[4][VW];
        #pragma unroll
        for (int u = 0; u < 4; ++u) {
          cj[u] = u < rem ? __ldg(colidx + e + u) : 0;
          vj[u] = u < rem ? __ldg(values + e + u) : T(0);
        }
        #pragma unroll
        for (int u = 0; u < 4; ++u)
          if (u < rem) ppr_ld<T, VW>(xo + (size_t)cj[u] * KT + c, xj[u]);
        #pragma unroll
        for (int u = 0; u < 4; ++u)
          if (u < rem)
            #pragma unroll
            for (int q = 0; q < VW; ++q) acc[q] = fma(vj[u], xj[u][q], acc[q]);
      }
    }
    if (it.w >= 0) {
      ppr_st<T, VW>(p.chunks + ((size_t)tl * p.slots + it.w) * KT + c, acc);
    } else {
      PprRowIn<T, VW, AA> in;
      ppr_row_in<T, VW, AA>(in, it.x, KT, c, pc, xo, seeds, p.dmask, rhs, ring);
      ppr_emit<T, VW, AA>(it.x, KT, c, acc, pc, in, xn, p.beta, rhs != nullptr, ring, res, dm, dots);
    }
    it = nx;
  }
  double part[NV][VW];
  ppr_gather_parts<T, VW, NV, AA>(res, dm, dots, part);
  block_columns<KT, VW, NV>(part, p.partials + (size_t)tl * p.nparts * KT * NV, blockIdx.x);
}

// rows cut into chunks: crow[h] = (row, first slot), crow[n].y = total slots;
// the chunks' sums are added in order, eight loads in flight
template <typename T, int KT, bool AA>
__global__ void __launch_bounds__(256) ppr_fixup_kernel(const int2 *__restrict__ crow, int n_crow, int part_base,
                                                       const PprSweep<T> p) {
  const int tl = blockIdx.y;
  if (*(volatile const int *)&p.tile[tl].done) return;
  constexpr int VW = PprLanes<T, KT>::VW, G = PprLanes<T, KT>::G, NV = AA ? 5 : 2;
  const int c = (threadIdx.x & (G - 1)) * VW;
  const size_t off = (size_t)tl * p.n * KT;
  const T *xo = p.xo + off;
  const T *rhs = p.rhs ? p.rhs + off : nullptr;
  const PprRing<T> ring{AA ? p.ring.r0 + off : nullptr, AA ? p.ring.r1 + off : nullptr,
                        AA ? p.ring.r2 + off : nullptr};
  const T *chunks = p.chunks + (size_t)tl * p.slots * KT;
  PprCols<VW> pc;
  ppr_cols<VW, AA>(pc, c, p.col + tl * KT, p.inv_size + tl * KT, p.aa + tl * KT);
  const int64_t ng = ((int64_t)gridDim.x * blockDim.x) / G;
  T res[VW];
  double dm[VW];
  #pragma unroll
  for (int q = 0; q < VW; ++q) {
    res[q] = 0;
    dm[q] = 0;
  }
  __shared__ T dots[AA ? 3 * VW * 256 : 1];
  if (AA)
    for (int j = 0; j < 3 * VW; ++j) dots[j * 256 + threadIdx.x] = 0;
  for (int64_t g = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / G; g < n_crow; g += ng) {
    const int2 h = crow[g];
    const int end = crow[g + 1].y;
    PprRowIn<T, VW, AA> in;
    ppr_row_in<T, VW, AA>(in, h.x, KT, c, pc, xo, p.seeds + (size_t)tl * p.n, p.dmask, rhs, ring);
    T acc[VW];
    #pragma unroll
    for (int q = 0; q < VW; ++q) acc[q] = 0;
    for (int s = h.y; s < end; s += 8) {
      T v[8][VW];
      #pragma unroll
      for (int u = 0; u < 8; ++u)
        if (s + u < end) ppr_ld<T, VW>(chunks + (size_t)(s + u) * KT + c, v[u]);
      #pragma unroll
      for (int u = 0; u < 8; ++u)
        if (s + u < end)
          #pragma unroll
          for (int q = 0; q < VW; ++q) acc[q] += v[u][q];
    }
    ppr_emit<T, VW, AA>(h.x, KT, c, acc, pc, in, p.xn + off, p.beta, rhs != nullptr, ring, res, dm, dots);
  }
  double part[NV][VW];
  ppr_gather_parts<T, VW, NV, AA>(res, dm, dots, part);
  block_columns<KT, VW, NV>(part, p.partials + (size_t)tl * p.nparts * KT * NV, part_base + blockIdx.x);
}

// per column: sum the parts in order, advance the column, then the tile.
// Accelerated: the new output's term and residual dots enter the column's
// history and the weights of the next input are solved (aa_coefficients); a
// column that stops takes its last output as it is.
// kPprFin blocks a tile (blockIdx.y): block b takes the parts b, b + kPprFin,
// ... (its warps every 32nd of them in order, the lanes a part's KT * NV values
// together, then the warps in order), and the block that arrives last adds the
// blocks' sums in order and, one thread per column, advances the columns.  One
// block for all parts took 55 us for the 1824 parts of a 32-vector tile.
constexpr int kPprFin = 16;
template <int KT, bool AA>
__global__ void __launch_bounds__(1024) ppr_finalize_kernel(const double *__restrict__ all_partials, size_t tile_parts,
                                                           int nparts, double *fin, unsigned *arrived, ColCtl *cols,
                                                           ColAa *aas, TileCtl *tiles, double beta, double cst,
                                                           int max_iter, int k, int first) {
  constexpr int NV = AA ? 5 : 2, W = KT * NV, PER = (W + 31) / 32;
  __shared__ double sh[32][W];
  __shared__ int active, last;
  const int tl = blockIdx.y;
  TileCtl *tile = tiles + tl;
  ColCtl *col = cols + tl * KT;
  ColAa *aa = aas + tl * KT;
  if (*(volatile int *)&tile->done) {
    if (threadIdx.x == 0 && blockIdx.x == 0) tile->ran = 0;
    return;
  }
  if (threadIdx.x == 0) active = 0;
  const double *partials = all_partials + (size_t)tl * tile_parts * W;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double a[PER];
  #pragma unroll
  for (int i = 0; i < PER; ++i) a[i] = 0;
  #pragma unroll 4
  for (int p = blockIdx.x + kPprFin * warp; p < nparts; p += 32 * kPprFin)
    #pragma unroll
    for (int i = 0; i < PER; ++i)
      if (lane + 32 * i < W) a[i] += partials[(size_t)p * W + lane + 32 * i];
  #pragma unroll
  for (int i = 0; i < PER; ++i)
    if (lane + 32 * i < W) sh[warp][lane + 32 * i] = a[i];
  __syncthreads();
  double *mine = fin + (size_t)tl * kPprFin * W;
  if (threadIdx.x < W) {
    double t = 0;
    for (int w = 0; w < 32; ++w) t += sh[w][threadIdx.x];
    __stcg(mine + (size_t)blockIdx.x * W + threadIdx.x, t);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicInc(arrived + tl, kPprFin - 1) == kPprFin - 1;  // back to 0 with the last
    __threadfence();
  }
  __syncthreads();
  if (!last) return;
  if (threadIdx.x < W) {
    double b[kPprFin], t = 0;
    #pragma unroll
    for (int w = 0; w < kPprFin; ++w) b[w] = __ldcg(mine + (size_t)w * W + threadIdx.x);
    #pragma unroll
    for (int w = 0; w < kPprFin; ++w) t += b[w];
    sh[0][threadIdx.x] = t;
  }
  __syncthreads();
  const int c = threadIdx.x;
  double v[NV];
  if (c < KT)
    #pragma unroll
    for (int j = 0; j < NV; ++j) v[j] = sh[0][c * NV + j];
  if (c < KT) {
    const double r = v[0], d = v[1];
    ColCtl &cc = col[c];
    if (first) {
      cc.add = beta * d + cst;  // initial vector: only the dangling mass is new
    } else if (!cc.done) {
      cc.iter += 1;
      cc.resid = r;
      cc.add = beta * d + cst;
      cc.done = r < cc.tol || cc.iter >= max_iter;
      if constexpr (AA) {
        ColAa &st = aa[c];
        st.add[2] = st.add[1];
        st.add[1] = st.add[0];
        st.add[0] = beta * d + cst;
        aa_gram_push(st.gram, v[2], v[3], v[4]);
        st.hist = min(st.hist + 1, 3);
        if (cc.done) {
          st.coef[0] = 1.0;
          st.coef[1] = st.coef[2] = 0.0;
          st.m = 0;
        } else {
          st.m = aa_coefficients(st.gram, st.hist - 1, st.coef);
          double add = st.coef[0] * st.add[0];
          if (st.m >= 1) add += st.coef[1] * st.add[1];
          if (st.m >= 2) add += st.coef[2] * st.add[2];
          cc.add = add;
        }
      }
    } else {
      cc.add = beta * d + cst;
    }
    if (tl * KT + c < k && !cc.done) atomicOr(&active, 1);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (!first) tile->iter += 1;
    tile->done = active == 0;
    tile->ran = 1;
  }
}

// accelerated: x = c0 g0 + c1 g1 + c2 g2 per column (g0 the newest output;
// only the terms in use are read), after every sweep that ran on the tile
// (also the one that stopped its last vector: x then takes its outputs)
template <typename T, int KT>
__global__ void __launch_bounds__(256) ppr_combine_kernel(int n, const T *__restrict__ g0,
                                                         const T *__restrict__ g1, const T *__restrict__ g2,
                                                         T *__restrict__ x, const ColAa *__restrict__ aas,
                                                         const TileCtl *tiles) {
  const int tl = blockIdx.y;
  if (!*(volatile const int *)&tiles[tl].ran) return;
  const ColAa *aa = aas + tl * KT;
  const size_t off = (size_t)tl * n * KT;
  constexpr int VW = PprLanes<T, KT>::VW, G = PprLanes<T, KT>::G;
  const int c = (threadIdx.x & (G - 1)) * VW;
  T c0[VW], c1[VW], c2[VW];
  int m[VW], mm = 0;
  #pragma unroll
  for (int q = 0; q < VW; ++q) {
    const ColAa &st = aa[c + q];
    c0[q] = (T)st.coef[0];
    c1[q] = (T)st.coef[1];
    c2[q] = (T)st.coef[2];
    m[q] = st.m;
    mm = max(mm, m[q]);
  }
  const int64_t ng = ((int64_t)gridDim.x * blockDim.x) / G;
  for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / G; i < n; i += ng) {
    const size_t at = off + (size_t)i * KT + c;
    T a[VW], b[VW], e[VW], v[VW];
    ppr_ld<T, VW>(g0 + at, a);
    if (mm >= 1) ppr_ld<T, VW>(g1 + at, b);
    if (mm >= 2) ppr_ld<T, VW>(g2 + at, e);
    #pragma unroll
    for (int q = 0; q < VW; ++q) {
      v[q] = c0[q] * a[q];
      if (m[q] >= 1) v[q] = fma(c1[q], b[q], v[q]);
      if (m[q] >= 2) v[q] = fma(c2[q], e[q], v[q]);
    }
    ppr_st<T, VW>(x + at, v);
  }
}

// x0 = v (seeds), dangling mass of x0 per column (partials of NV values per
// column, the others 0)
template <typename T, int KT, int NV>
__global__ void __launch_bounds__(256) ppr_init_kernel(int n, const unsigned *__restrict__ seeds,
                                                      const unsigned char *__restrict__ dmask,
                                                      const double *__restrict__ inv_size, T *__restrict__ x,
                                                      double *partials) {
  const int c = threadIdx.x & (KT - 1);
  const int64_t ng = ((int64_t)gridDim.x * blockDim.x) / KT;
  double part[NV][1] = {};
  for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / KT; i < n; i += ng) {
    const T v = ((seeds[i] >> c) & 1u) ? (T)inv_size[c] : T(0);
    x[(size_t)i * KT + c] = v;
    if (dmask[i]) part[1][0] += (double)v;
  }
  block_columns<KT, 1, NV>(part, partials, blockIdx.x);
}

// x (one tile) from FP64 vectors in the original labels: vector vec[c] of
// src (src + vec[c] * n) at tile row newid[u] (u when not relabelled);
// columns with vec[c] < 0 get 0.  With partials: the dangling mass per column.
template <typename T, int KT, int NV>
__global__ void __launch_bounds__(256) ppr_load_kernel(int n, const double *__restrict__ src,
                                                      const int *__restrict__ vec, const int *__restrict__ newid,
                                                      const unsigned char *__restrict__ dmask, T *__restrict__ x,
                                                      double *partials) {
  const int c = threadIdx.x & (KT - 1);
  const int64_t ng = ((int64_t)gridDim.x * blockDim.x) / KT;
  const int v = vec[c];
  double part[NV][1] = {};
  for (int64_t u = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / KT; u < n; u += ng) {
    const int i = newid ? newid[u] : (int)u;
    const T val = v >= 0 ? (T)src[(size_t)v * n + u] : T(0);
    x[(size_t)i * KT + c] = val;
    if (partials && dmask[i]) part[1][0] += (double)val;
  }
  if (partials) block_columns<KT, 1, NV>(part, partials, blockIdx.x);
}

// out[v_j * n + u] = column c_j of a tile at row map(u), as FP64, for the
// cnt (column, vector) pairs of a list
struct PprPicks {
  int cnt;
  int col[32], vec[32];
};
template <typename T, int KT>
__global__ void ppr_pick_kernel(const T *__restrict__ x, int n, const int *__restrict__ newid, PprPicks pk,
                                double *__restrict__ out) {
  const int64_t total = (int64_t)n * pk.cnt;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int j = (int)(t / n), u = (int)(t % n);
    const int i = newid ? newid[u] : u;
    out[(size_t)pk.vec[j] * n + u] = (double)x[(size_t)i * KT + pk.col[j]];
  }
}

// repacked layout: slot s of the new tiles takes old slot map[s] (-1: zero)
template <typename T, int KT>
__global__ void ppr_move_kernel(const T *__restrict__ src, T *__restrict__ dst, int n, const int *__restrict__ map,
                                int new_tiles) {
  const int64_t total = (int64_t)new_tiles * n * KT;
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < total; q += (int64_t)gridDim.x * blockDim.x) {
    const int c = (int)(q % KT);
    const int64_t ti = q / KT;
    const int i = (int)(ti % n), t = (int)(ti / n);
    const int from = map[t * KT + c];
    dst[q] = from < 0 ? T(0) : src[((size_t)(from / KT) * n + i) * KT + (from % KT)];
  }
}

// seeds[(slot / KT) * n + node] |= bit (slot % KT) for the (slot, node) pairs
// of the seed sets (the array zeroed before)
template <int KT>
__global__ void ppr_seed_bits_kernel(unsigned *seeds, int n, const int2 *__restrict__ pairs, int npairs) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < npairs; i += gridDim.x * blockDim.x) {
    const int2 q = pairs[i];
    atomicOr(seeds + (size_t)(q.x / KT) * n + q.y, 1u << (q.x % KT));
  }
}

// Device memory kept with the handle between solves (allocating and freeing a
// solve's two dozen buffers took a third of a 64-vector solve on R-MAT 2^17:
// six FP32 and FP64 solves of a refined one).  One solve holds it at a time,
// others allocate their own; more than kPprKeepBytes is given back at the end
// of the solve, the rest with the handle.
constexpr size_t kPprKeepBytes = (size_t)512 << 20;
struct PprMemory {
  std::mutex busy;
  char *base = nullptr;
  size_t bytes = 0;
};
// The buffers of one solve, cut from one allocation: add() the requests, then
// get(); released (after the work that uses it) by the destructor.
class PprBuffers {
 public:
  PprBuffers(PprMemory *kept, cudaStream_t s) : kept_(kept), s_(s) {}
  ~PprBuffers() {
    if (!base_) return;
    cudaStreamSynchronize(s_);
    if (!mine_) {
      if (kept_->bytes > kPprKeepBytes) drop();
      kept_->busy.unlock();
    } else {
      cudaFree(base_);
    }
  }
  template <typename T> void add(T **p, size_t bytes) {
    req_.push_back({reinterpret_cast<void **>(p), (bytes + 255) / 256 * 256 + 256});
  }
  tbsla_status_t get() {
    size_t total = 0;
    for (auto &r : req_) total += r.second;
    mine_ = !kept_->busy.try_lock();
    cudaError_t e = cudaSuccess;
    if (mine_) {
      e = cudaMalloc((void **)&base_, total);
    } else {
      if (kept_->bytes < total) {
        drop();
        e = cudaMalloc((void **)&kept_->base, total);
        if (e == cudaSuccess) kept_->bytes = total;
        else kept_->base = nullptr;
      }
      base_ = kept_->base;
      if (e != cudaSuccess) kept_->busy.unlock();
    }
    if (e != cudaSuccess) {
      cudaGetLastError();
      base_ = nullptr;
      return fail(TBSLA_ERR_OOM, "batched PageRank buffers (%zu bytes)", total);
    }
    char *p = base_;
    for (auto &r : req_) {
      *r.first = p;
      p += r.second;
    }
    return TBSLA_OK;
  }

 private:
  void drop() {
    if (kept_->base) cudaFree(kept_->base);
    kept_->base = nullptr;
    kept_->bytes = 0;
  }
  PprMemory *kept_;
  cudaStream_t s_;
  char *base_ = nullptr;
  bool mine_ = false;
  std::vector<std::pair<void **, size_t>> req_;
};

// The work list of a handle's batched sweeps in decreasing length: rows, and
// rows longer than a chunk cut into chunks; built once (it depends on the row
// structure only) and kept on the handle.  A chunk is walked by one row group,
// so it is a 16384th of the entries, 64 to 512: on small graphs a long chunk
// outlasts the sweep (R-MAT 2^17, 32 FP32 vectors: 179 us a sweep with chunks
// of 512 entries), on large ones short chunks only cost partial sums.
struct PprPlan {
  PprMemory solve, refine;  // buffers of a solve, and of the refinement around it
  int4 *items = nullptr;  // (row, begin, end, chunk slot or -1)
  int2 *crow = nullptr;   // chunked rows: (row, first slot); crow[n_crow].y = slots
  int n_items = 0, n_crow = 0, slots = 0;
};
void ppr_plan_free(void *q) {
  PprPlan *P = static_cast<PprPlan *>(q);
  if (P->solve.base) cudaFree(P->solve.base);
  if (P->refine.base) cudaFree(P->refine.base);
  if (P->items) cudaFree(P->items);
  if (P->crow) cudaFree(P->crow);
  delete P;
}
tbsla_status_t ppr_plan(const tbsla_matrix *Mc, PprPlan **out) {
  tbsla_matrix *M = const_cast<tbsla_matrix *>(Mc);
  std::lock_guard<std::mutex> lk(M->first_use);
  if (M->ppr_plan) {
    *out = static_cast<PprPlan *>(M->ppr_plan);
    return TBSLA_OK;
  }
  const int n = M->n_row;
  std::vector<int> rp((size_t)n + 1);
  TB_CUDA(cudaMemcpy(rp.data(), M->idx0, ((size_t)n + 1) * sizeof(int), cudaMemcpyDeviceToHost));
  int chunk = kPprChunkMin;
  while (chunk < kPprChunkMax && (int64_t)chunk * 2 * 16384 <= M->stored) chunk *= 2;
  std::vector<int4> items;
  std::vector<int2> crow;
  int slots = 0;
  items.reserve((size_t)n);
  for (int r = 0; r < n; ++r) {
    const int a = rp[(size_t)r], b = rp[(size_t)r + 1];
    if (b - a <= chunk) {
      items.push_back(make_int4(r, a, b, -1));
      continue;
    }
    crow.push_back(make_int2(r, slots));
    for (int e = a; e < b; e += chunk) items.push_back(make_int4(r, e, std::min(e + chunk, b), slots++));
  }
  // decreasing length, equal lengths in row order (a counting sort)
  {
    std::vector<size_t> at((size_t)chunk + 2, 0);
    for (const int4 &q : items) ++at[(size_t)(chunk - (q.z - q.y)) + 1];
    for (size_t l = 1; l < at.size(); ++l) at[l] += at[l - 1];
    std::vector<int4> sorted(items.size());
    for (const int4 &q : items) sorted[at[(size_t)(chunk - (q.z - q.y))]++] = q;
    items.swap(sorted);
  }
  PprPlan *P = new PprPlan;
  P->n_items = (int)items.size();
  P->n_crow = (int)crow.size();
  P->slots = slots;
  crow.push_back(make_int2(-1, slots));
  if (cudaMalloc((void **)&P->items, std::max<size_t>(items.size(), 1) * sizeof(int4)) != cudaSuccess ||
      cudaMalloc((void **)&P->crow, crow.size() * sizeof(int2)) != cudaSuccess) {
    cudaGetLastError();
    ppr_plan_free(P);
    return fail(TBSLA_ERR_OOM, "batched PageRank work list");
  }
  if ((!items.empty() &&
       cudaMemcpy(P->items, items.data(), items.size() * sizeof(int4), cudaMemcpyHostToDevice) != cudaSuccess) ||
      cudaMemcpy(P->crow, crow.data(), crow.size() * sizeof(int2), cudaMemcpyHostToDevice) != cudaSuccess) {
    ppr_plan_free(P);
    return fail(TBSLA_ERR_CUDA, "batched PageRank work list upload");
  }
  M->ppr_plan = P;
  M->ppr_plan_free = ppr_plan_free;
  *out = P;
  return TBSLA_OK;
}

// Accelerated repacking, in place: destination tile t of buf takes, per
// column c, old slot map[c] (-1: zero).  The live vectors keep their order,
// so every source of tile t lies in tile t or later; with the destination
// tiles done in increasing order (one launch each) and the lanes of a warp
// reading all their rows' sources before any of them writes (a row's sources
// and destinations are in the same row, one warp's), nothing is overwritten
// before it is read.
template <typename T, int KT>
__global__ void __launch_bounds__(256) ppr_compact_kernel(T *buf, int n, const int *__restrict__ map, int t) {
  constexpr int VW = PprLanes<T, KT>::VW, G = PprLanes<T, KT>::G;
  const int c = (threadIdx.x & (G - 1)) * VW;
  int from[VW];
  #pragma unroll
  for (int q = 0; q < VW; ++q) from[q] = map[c + q];
  const int64_t ng = ((int64_t)gridDim.x * blockDim.x) / G;
  // warp-uniform loop: the warp's first row, then its lanes' rows
  for (int64_t i0 = ((int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31)) / G; i0 < n; i0 += ng) {
    const int64_t i = i0 + (threadIdx.x & 31) / G;
    T v[VW];
    if (i < n) {
      #pragma unroll
      for (int q = 0; q < VW; ++q)
        v[q] = from[q] < 0 ? T(0) : buf[((size_t)(from[q] / KT) * n + i) * KT + (from[q] % KT)];
    }
    __syncwarp();
    if (i < n) ppr_st<T, VW>(buf + ((size_t)t * n + i) * KT + c, v);
  }
}

// Options of one batched solve: by default x0 = v_c and the teleport form
// x = beta A x + (beta d.x + 1 - beta) v_c.  A defect-correction solve passes
// x0 = rhs = r_c and cst = 0: e = beta A e + beta (d.e) v_c + r_c.
struct RunOpts {
  const double *x0 = nullptr;   // start: vector c at x0 + src(c) * n (original labels), FP64
  const double *rhs = nullptr;  // added to every sweep: rhs + src(c) * n
  const int *src = nullptr;     // host: column of x0 / rhs for vector c (NULL: c)
  double cst = -1.0;            // the constant of the teleport term (< 0: 1 - beta)
  const double *tol = nullptr;  // host: stopping threshold per vector (NULL: p->tol)
};

// One batched solve in tiles of KT vectors; AA: Anderson-accelerated
// (p->accel).  Plain sweeps ping-pong between two iterate buffers per tile;
// accelerated ones read the iterate x, write the output g and residual r to
// slot j % 3 of their rings (j counting the solve's sweeps), and the
// combination of the last three outputs becomes the next x.
template <typename T, int KT, bool AA>
tbsla_status_t run_tiles_impl(const tbsla_matrix *M, const int *newid_dev, const std::vector<int> *newid_host,
                              const tbsla_pagerank_params_t *p, int k, const int *nodes, const int *offsets,
                              double *d_out, int *iters_out, double *resid_out, cudaStream_t s, const RunOpts &opt) {
  constexpr int NV = AA ? 5 : 2;
  constexpr int G = PprLanes<T, KT>::G;
  const int n = M->n_row;
  const T *values = static_cast<const T *>(M->values[std::is_same<T, double>::value ? 0 : 1]);
  TB_CHECK(values, "the matrix lacks the %s value store", std::is_same<T, double>::value ? "F64" : "F32");
  const int tiles = (k + KT - 1) / KT;
  PprPlan *plan = nullptr;
  TB_TRY(ppr_plan(M, &plan));
  const int n_crow = plan->n_crow, slots = plan->slots;
  // seeds: bit c of seeds[t*n + i] = row i is a seed of vector t*KT + c, set
  // on the device from the (slot, node) pairs
  std::vector<int2> pairs;
  std::vector<double> inv((size_t)tiles * KT, 0.0);
  std::vector<std::vector<int>> seed_sets((size_t)k);  // per vector, in the matrix's labels
  for (int c = 0; c < k; ++c) {
    const int b = offsets[c], e = offsets[c + 1];
    TB_CHECK(e > b, "vector %d has an empty seed set", c);
    std::vector<int> &dist = seed_sets[(size_t)c];
    for (int q = b; q < e; ++q) {
      int v = nodes[q];
      TB_CHECK(v >= 0 && v < n, "seed %d of vector %d outside [0, %d)", v, c, n);
      if (newid_host) v = (*newid_host)[(size_t)v];
      dist.push_back(v);
    }
    std::sort(dist.begin(), dist.end());
    dist.erase(std::unique(dist.begin(), dist.end()), dist.end());
    for (int v : dist) pairs.push_back(make_int2(c, v));
    inv[(size_t)c] = 1.0 / (double)dist.size();
  }
  // the sweep grid of a tile: the blocks that fit on the GPU at once (the items
  // are dealt in decreasing length, so one wave is even)
  int sms = 0, per_sm = 0;
  TB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, M->device));
  TB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ppr_spmm_kernel<T, KT, AA>, 256, 0));
  const int grid_mm = std::max(1, sms * std::max(per_sm, 1));
  const int grid_fx = std::max(1, std::min((n_crow * G + 255) / 256, sms * 4));
  const int grid_in = 152 * 4;
  const int grid_vec = 152 * 8;  // streaming passes over a tile (combine, compaction)
  const int nparts = std::max(grid_mm + grid_fx, grid_in);
  // device buffers
  const size_t xbytes = (size_t)n * KT * sizeof(T);
  T *x[2] = {nullptr, nullptr};
  T *g_ring[3] = {nullptr, nullptr, nullptr}, *r_ring[3] = {nullptr, nullptr, nullptr};
  T *chunk = nullptr;
  unsigned *d_seeds = nullptr;
  int2 *d_pairs = nullptr;
  unsigned char *dmask = nullptr;
  int *d_zeros = nullptr;
  double *d_inv = nullptr, *partials = nullptr, *fin = nullptr;
  unsigned *arrived = nullptr;
  ColCtl *d_col = nullptr;
  ColAa *d_aa = nullptr;
  TileCtl *d_tile = nullptr;
  T *rhs_t[2] = {nullptr, nullptr};  // the right-hand side in the tiles' layout (ping-pong for repacking)
  int *d_vec = nullptr;              // per slot: the column of x0 / rhs it holds, or -1
  char *d_ctl = nullptr;  // tile, column and Anderson state, one after another: one copy reads them
  int *d_map = nullptr;
  PprBuffers buffers(&plan->solve, s);
  auto alloc = [&](void **ptr, size_t bytes) { buffers.add(ptr, bytes); };
  alloc((void **)&x[0], (size_t)tiles * xbytes);
  if (AA) {
    for (int j = 0; j < 3; ++j) {
      alloc((void **)&g_ring[j], (size_t)tiles * xbytes);
      alloc((void **)&r_ring[j], (size_t)tiles * xbytes);
    }
  } else {
    alloc((void **)&x[1], (size_t)tiles * xbytes);
  }
  alloc((void **)&chunk, (size_t)tiles * std::max(slots, 1) * KT * sizeof(T));
  alloc((void **)&fin, (size_t)tiles * kPprFin * KT * NV * sizeof(double));
  alloc((void **)&arrived, (size_t)tiles * sizeof(unsigned));
  alloc((void **)&d_seeds, (size_t)tiles * n * sizeof(unsigned));
  alloc((void **)&d_pairs, pairs.size() * sizeof(int2));
  alloc((void **)&dmask, (size_t)n);
  alloc((void **)&d_zeros, sizeof(int));
  alloc((void **)&d_inv, inv.size() * sizeof(double));
  alloc((void **)&partials, (size_t)tiles * nparts * KT * NV * sizeof(double));
  const size_t col_at = (size_t)tiles * sizeof(TileCtl), aa_at = col_at + (size_t)tiles * KT * sizeof(ColCtl);
  const size_t ctl_bytes = aa_at + (AA ? (size_t)tiles * KT * sizeof(ColAa) : 0);
  static_assert(sizeof(TileCtl) % 8 == 0 && sizeof(ColCtl) % 8 == 0, "the control arrays follow one another");
  alloc((void **)&d_ctl, aa_at + (size_t)tiles * KT * sizeof(ColAa));
  alloc((void **)&d_vec, (size_t)tiles * KT * sizeof(int));
  alloc((void **)&d_map, (size_t)tiles * KT * sizeof(int));
  if (opt.rhs) {
    alloc((void **)&rhs_t[0], (size_t)tiles * xbytes);
    if (!AA) alloc((void **)&rhs_t[1], (size_t)tiles * xbytes);
  }
  TB_TRY(buffers.get());
  d_tile = reinterpret_cast<TileCtl *>(d_ctl);
  d_col = reinterpret_cast<ColCtl *>(d_ctl + col_at);
  d_aa = reinterpret_cast<ColAa *>(d_ctl + aa_at);
  const double cst = opt.cst < 0 ? 1.0 - p->beta : opt.cst;
  auto src_col = [&](int v) { return v < 0 ? -1 : opt.src ? opt.src[v] : v; };
  std::vector<ColCtl> hcol((size_t)tiles * KT);
  std::vector<int> hvec((size_t)tiles * KT, -1);
  for (int c = 0; c < tiles * KT; ++c) {
    // padding columns start stopped
    hcol[(size_t)c] = ColCtl{0.0, 0.0, c < k && opt.tol ? opt.tol[c] : p->tol, 0, c >= k ? 1 : 0};
    hvec[(size_t)c] = src_col(c < k ? c : -1);
  }
  // no history; the plain step
  ColAa aa0;
  std::memset(&aa0, 0, sizeof(aa0));
  aa0.coef[0] = 1.0;
  std::vector<ColAa> haa((size_t)tiles * KT, aa0);
  std::vector<TileCtl> htile((size_t)tiles, TileCtl{0, 0, 0, 0});
  if (p->max_iter == 0)
    for (auto &tc : htile) tc.done = 1;
  cudaError_t e = cudaSuccess;
  auto up = [&](void *d, const void *h, size_t b) {
    if (e == cudaSuccess && b) e = cudaMemcpyAsync(d, h, b, cudaMemcpyHostToDevice, s);
  };
  up(d_pairs, pairs.data(), pairs.size() * sizeof(int2));
  if (e == cudaSuccess) e = cudaMemsetAsync(arrived, 0, (size_t)tiles * sizeof(unsigned), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(d_seeds, 0, (size_t)tiles * n * sizeof(unsigned), s);
  if (e == cudaSuccess)
    ppr_seed_bits_kernel<KT><<<152, 256, 0, s>>>(d_seeds, n, d_pairs, (int)pairs.size());
  up(d_inv, inv.data(), inv.size() * sizeof(double));
  up(d_col, hcol.data(), hcol.size() * sizeof(ColCtl));
  up(d_aa, haa.data(), haa.size() * sizeof(ColAa));
  up(d_tile, htile.data(), htile.size() * sizeof(TileCtl));
  up(d_vec, hvec.data(), hvec.size() * sizeof(int));
  if (e != cudaSuccess) return fail(TBSLA_ERR_CUDA, "batched PageRank upload: %s", cudaGetErrorString(e));
  TB_TRY(column_mask(const_cast<tbsla_matrix *>(M), values, dmask, d_zeros, s));
  const double beta = p->beta;
  for (int t = 0; t < tiles; ++t) {
    double *pt = partials + (size_t)t * nparts * KT * NV;
    if (opt.x0)
      ppr_load_kernel<T, KT, NV><<<grid_in, 256, 0, s>>>(n, opt.x0, d_vec + (size_t)t * KT, newid_dev, dmask,
                                                         x[0] + (size_t)t * n * KT, pt);
    else
      ppr_init_kernel<T, KT, NV><<<grid_in, 256, 0, s>>>(n, d_seeds + (size_t)t * n, dmask,
                                                         d_inv + (size_t)t * KT, x[0] + (size_t)t * n * KT, pt);
    if (opt.rhs)
      ppr_load_kernel<T, KT, NV><<<grid_in, 256, 0, s>>>(n, opt.rhs, d_vec + (size_t)t * KT, newid_dev, dmask,
                                                         rhs_t[0] + (size_t)t * n * KT, nullptr);
  }
  // launches over the tiles of a layout (blockIdx.y, at most kTilesPerLaunch)
  constexpr int kTilesPerLaunch = 65535;
  auto finalize = [&](int count, int parts, int first) {
    for (int t = 0; t < count; t += kTilesPerLaunch)
      ppr_finalize_kernel<KT, AA><<<dim3(kPprFin, std::min(kTilesPerLaunch, count - t)), 1024, 0, s>>>(
          partials + (size_t)t * nparts * KT * NV, (size_t)nparts, parts, fin + (size_t)t * kPprFin * KT * NV,
          arrived + t, d_col + (size_t)t * KT, d_aa + (size_t)t * KT, d_tile + t, beta, cst, p->max_iter,
          first ? k - t * KT : count * KT, first);
  };
  finalize(tiles, grid_in, 1);
  int rbase = 0;  // rhs_t[rbase] holds the current layout's right-hand side
  if (cudaGetLastError() != cudaSuccess) return fail(TBSLA_ERR_CUDA, "batched PageRank init");
  // Sweeps in sets of K on every tile of the current layout (stopped tiles
  // return at once).  After each set the vectors that stopped are written
  // out and dropped; when the live vectors fit in fewer tiles they are
  // repacked (compaction), so a tile never keeps sweeping for one slow
  // vector while its other lanes idle.  All tiles of a layout sweep in step:
  // plain, the layout's iterates start in x[base] and sweep j reads
  // x[(base+j)&1]; accelerated, sweep number gk of the solve writes ring slot
  // gk % 3.
  // sweeps per look of the host (4: R-MAT 2^22, 256 vectors, 3-9 % faster than 8)
  const int K = std::min(p->check_every > 0 ? p->check_every : 4, std::max(p->max_iter, 1));
  int cur_tiles = tiles, base = 0;
  int64_t gk = 0;
  std::vector<int> slot_vec((size_t)tiles * KT, -1);  // vector in each slot, -1 for none
  for (int c = 0; c < k; ++c) slot_vec[(size_t)c] = c;
  std::vector<TileCtl> htc((size_t)tiles);
  std::vector<ColCtl> hcc((size_t)tiles * KT);
  std::vector<ColAa> hca((size_t)tiles * KT);
  std::vector<char> hctl(ctl_bytes);
  int phase = 0;
  const size_t tstride = (size_t)n * KT;
  while (true) {
    for (int k2 = 0; k2 < K; ++k2, ++phase, ++gk) {
      const int w = (int)(gk % 3), w1 = (int)((gk + 2) % 3), w2 = (int)((gk + 1) % 3);
      for (int t = 0; t < cur_tiles; t += kTilesPerLaunch) {
        const unsigned count = (unsigned)std::min(kTilesPerLaunch, cur_tiles - t);
        const size_t off = (size_t)t * tstride;
        PprSweep<T> sw;
        sw.xo = AA ? x[0] + off : x[(base + phase) & 1] + off;
        sw.xn = AA ? g_ring[w] + off : x[(base + phase + 1) & 1] + off;
        sw.ring = PprRing<T>{AA ? r_ring[w] + off : nullptr, AA ? r_ring[w1] + off : nullptr,
                             AA ? r_ring[w2] + off : nullptr};
        sw.rhs = opt.rhs ? rhs_t[rbase] + off : nullptr;
        sw.seeds = d_seeds + (size_t)t * n;
        sw.dmask = dmask;
        sw.col = d_col + (size_t)t * KT;
        sw.aa = d_aa + (size_t)t * KT;
        sw.inv_size = d_inv + (size_t)t * KT;
        sw.chunks = chunk + (size_t)t * slots * KT;
        sw.partials = partials + (size_t)t * nparts * KT * NV;
        sw.tile = d_tile + t;
        sw.beta = beta;
        sw.n = n;
        sw.slots = slots;
        sw.nparts = nparts;
        ppr_spmm_kernel<T, KT, AA><<<dim3(grid_mm, count), 256, 0, s>>>(plan->items, plan->n_items, M->idx1, values, sw);
        if (n_crow)
          ppr_fixup_kernel<T, KT, AA><<<dim3(grid_fx, count), 256, 0, s>>>(plan->crow, n_crow, grid_mm, sw);
      }
      finalize(cur_tiles, n_crow ? grid_mm + grid_fx : grid_mm, 0);
      if (AA)
        for (int t = 0; t < cur_tiles; t += kTilesPerLaunch) {
          const size_t off = (size_t)t * tstride;
          ppr_combine_kernel<T, KT><<<dim3(grid_vec, std::min(kTilesPerLaunch, cur_tiles - t)), 256, 0, s>>>(
              n, g_ring[w] + off, g_ring[w1] + off, g_ring[w2] + off, x[0] + off, d_aa + (size_t)t * KT, d_tile + t);
        }
    }
    if (cudaMemcpyAsync(hctl.data(), d_ctl, ctl_bytes, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
      return fail(TBSLA_ERR_CUDA, "batched PageRank sweeps failed");
    std::memcpy(htc.data(), hctl.data(), (size_t)cur_tiles * sizeof(TileCtl));
    std::memcpy(hcc.data(), hctl.data() + col_at, (size_t)cur_tiles * KT * sizeof(ColCtl));
    if (AA) std::memcpy(hca.data(), hctl.data() + aa_at, (size_t)cur_tiles * KT * sizeof(ColAa));
    // write out and drop the vectors that stopped (a stopped vector is
    // frozen: plain, its tile's last iterate, x[(base + tile iter) & 1],
    // holds it; accelerated, x; a stopped tile's vectors have all stopped,
    // or max_iter is 0)
    int live = 0, busy = 0;
    for (int t = 0; t < cur_tiles; ++t) {
      PprPicks pk;
      pk.cnt = 0;
      for (int c = 0; c < KT; ++c) {
        const int v = slot_vec[(size_t)t * KT + c];
        if (v < 0) continue;
        const ColCtl &cc = hcc[(size_t)t * KT + c];
        if (cc.done || htc[(size_t)t].done) {
          pk.col[pk.cnt] = c;
          pk.vec[pk.cnt++] = v;
          if (iters_out) iters_out[v] = cc.iter;
          if (resid_out) resid_out[v] = cc.resid;
          slot_vec[(size_t)t * KT + c] = -1;
        } else {
          ++live;
        }
      }
      if (pk.cnt) {
        const T *xf = (AA ? x[0] : x[(base + htc[(size_t)t].iter) & 1]) + (size_t)t * tstride;
        ppr_pick_kernel<T, KT><<<152 * 8, 256, 0, s>>>(xf, n, newid_dev, pk, d_out);
      }
      busy += !htc[(size_t)t].done;
    }
    if (cudaGetLastError() != cudaSuccess) return fail(TBSLA_ERR_CUDA, "batched PageRank results");
    if (live == 0) break;
    const int need = (live + KT - 1) / KT;
    if (need < busy) {
      // repack the live vectors into `need` tiles (every live tile has run all
      // `phase` sweeps of the layout): plain, their iterates (in
      // x[(base+phase)&1]) move to the other buffer, which becomes the new
      // layout's start; accelerated, the iterates, the rings and the
      // right-hand side are compacted in place
      std::vector<int> map((size_t)need * KT, -1), nvec((size_t)need * KT, -1);
      std::vector<int2> npairs;
      std::vector<double> ninv((size_t)need * KT, 0.0);
      std::vector<ColCtl> ncol((size_t)need * KT);
      std::vector<ColAa> naa((size_t)need * KT, aa0);
      int q = 0;
      for (int t = 0; t < cur_tiles; ++t)
        for (int c = 0; c < KT; ++c) {
          const int v = slot_vec[(size_t)t * KT + c];
          if (v < 0) continue;
          map[(size_t)q] = t * KT + c;
          nvec[(size_t)q] = v;
          ncol[(size_t)q] = hcc[(size_t)t * KT + c];
          if (AA) naa[(size_t)q] = hca[(size_t)t * KT + c];
          ninv[(size_t)q] = inv[(size_t)t * KT + c];
          for (int u : seed_sets[(size_t)v]) npairs.push_back(make_int2(q, u));
          ++q;
        }
      for (size_t r = (size_t)q; r < ncol.size(); ++r) ncol[r] = ColCtl{0.0, 0.0, 0.0, 0, 1};
      std::vector<TileCtl> ntile((size_t)need, TileCtl{0, 0, 0, 0});
      up(d_map, map.data(), map.size() * sizeof(int));
      up(d_pairs, npairs.data(), npairs.size() * sizeof(int2));  // no more pairs than at the start
      if (e == cudaSuccess) e = cudaMemsetAsync(d_seeds, 0, (size_t)need * n * sizeof(unsigned), s);
      if (e == cudaSuccess)
        ppr_seed_bits_kernel<KT><<<152, 256, 0, s>>>(d_seeds, n, d_pairs, (int)npairs.size());
      up(d_inv, ninv.data(), ninv.size() * sizeof(double));
      up(d_col, ncol.data(), ncol.size() * sizeof(ColCtl));
      if (AA) up(d_aa, naa.data(), naa.size() * sizeof(ColAa));
      up(d_tile, ntile.data(), ntile.size() * sizeof(TileCtl));
      if (e != cudaSuccess) return fail(TBSLA_ERR_CUDA, "batched PageRank repack: %s", cudaGetErrorString(e));
      if (AA) {
        T *bufs[8] = {x[0], g_ring[0], g_ring[1], g_ring[2], r_ring[0], r_ring[1], r_ring[2], rhs_t[0]};
        for (int t = 0; t < need; ++t)
          for (T *b : bufs)
            if (b) ppr_compact_kernel<T, KT><<<grid_vec, 256, 0, s>>>(b, n, d_map + (size_t)t * KT, t);
      } else {
        const int src = (base + phase) & 1;
        ppr_move_kernel<T, KT><<<152 * 8, 256, 0, s>>>(x[src], x[src ^ 1], n, d_map, need);
        if (opt.rhs) {
          ppr_move_kernel<T, KT><<<152 * 8, 256, 0, s>>>(rhs_t[rbase], rhs_t[rbase ^ 1], n, d_map, need);
          rbase ^= 1;
        }
        base = src ^ 1;
      }
      if (cudaGetLastError() != cudaSuccess) return fail(TBSLA_ERR_CUDA, "batched PageRank repack");
      phase = 0;
      cur_tiles = need;
      slot_vec = nvec;
      inv = ninv;
    }
  }
  if (cudaStreamSynchronize(s) != cudaSuccess || cudaGetLastError() != cudaSuccess)
    return fail(TBSLA_ERR_CUDA, "batched PageRank results");
  return TBSLA_OK;
}

template <typename T, int KT>
tbsla_status_t run_tiles(const tbsla_matrix *M, const int *newid_dev, const std::vector<int> *newid_host,
                         const tbsla_pagerank_params_t *p, int k, const int *nodes, const int *offsets,
                         double *d_out, int *iters_out, double *resid_out, cudaStream_t s,
                         const RunOpts &opt = RunOpts()) {
  if (p->accel)
    return run_tiles_impl<T, KT, true>(M, newid_dev, newid_host, p, k, nodes, offsets, d_out, iters_out,
                                       resid_out, s, opt);
  return run_tiles_impl<T, KT, false>(M, newid_dev, newid_host, p, k, nodes, offsets, d_out, iters_out, resid_out,
                                      s, opt);
}

__global__ void ppr_sub_kernel(double *__restrict__ g, const double *__restrict__ x, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    g[i] -= x[i];
}
__global__ void ppr_add_kernel(double *__restrict__ x, const double *__restrict__ e, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    x[i] += e[i];
}

// FP32 sweeps with FP64 defect correction (tbsla_ppr_batched_refined):
// x = the FP32 solve; then rounds of r = G(x) - x by one FP64 sweep of every
// vector, stopping when every ||r_c||_1 < tol (the result is G(x)), else the
// FP32 correction solve e = beta A e + beta (d.e) v_c + r_c from e = r_c to
// ||e_j+1 - e_j||_1 < eta ||r_c||_1, and x += e.  Iterations: FP32 and FP64
// sweeps together.
constexpr double kRefineEta = 1e-3;       // inner tolerance relative to ||r_c||_1
constexpr double kRefineEtaAccel = 1e-4;  // the same for accelerated correction solves
constexpr double kF32SolveFloor = 1e-6; // the FP32 solve's stopping threshold at least this
constexpr int kRefineRounds = 8;

template <int KT>
tbsla_status_t run_refined(const tbsla_matrix *M, const int *nd, const std::vector<int> *nh,
                           const tbsla_pagerank_params_t *p, int k, const int *nodes, const int *offsets,
                           double *d_out, int *iters_out, double *resid_out, cudaStream_t s) {
  const int64_t n = M->n_row, total = n * k;
  std::vector<int> itot((size_t)k), it((size_t)k);
  std::vector<double> res((size_t)k, 0.0), tolc((size_t)k);
  tbsla_pagerank_params_t q = *p;
  q.tol = std::max(p->tol, kF32SolveFloor);
  TB_TRY((run_tiles<float, KT>(M, nd, nh, &q, k, nodes, offsets, d_out, itot.data(), nullptr, s)));
  double *g = nullptr, *e = nullptr;
  PprPlan *plan = nullptr;
  TB_TRY(ppr_plan(M, &plan));
  PprBuffers buffers(&plan->refine, s);
  buffers.add(&g, (size_t)total * sizeof(double));
  buffers.add(&e, (size_t)total * sizeof(double));
  TB_TRY(buffers.get());
  const int grid = 152 * 8;
  for (int round = 0;; ++round) {
    // r = G(x) - x: one FP64 sweep from x (the sweep's L1 change is ||r_c||_1)
    tbsla_pagerank_params_t q64 = *p;
    q64.max_iter = 1;
    q64.accel = 0;
    RunOpts o64;
    o64.x0 = d_out;
    TB_TRY((run_tiles<double, KT>(M, nd, nh, &q64, k, nodes, offsets, g, nullptr, res.data(), s, o64)));
    bool all = true;
    for (int c = 0; c < k; ++c) {
      itot[(size_t)c] += 1;
      all = all && res[(size_t)c] < p->tol;
    }
    if (all || round == kRefineRounds) {
      TB_CUDA(cudaMemcpyAsync(d_out, g, (size_t)total * sizeof(double), cudaMemcpyDeviceToDevice, s));
      break;
    }
    ppr_sub_kernel<<<grid, 256, 0, s>>>(g, d_out, total);
    TB_CUDA(cudaGetLastError());
    // the correction, only as far as each vector still needs it
    for (int c = 0; c < k; ++c)
      tolc[(size_t)c] = res[(size_t)c] < p->tol ? HUGE_VAL : (p->accel ? kRefineEtaAccel : kRefineEta) * res[(size_t)c];
    RunOpts oc;
    oc.x0 = g;
    oc.rhs = g;
    oc.cst = 0.0;
    oc.tol = tolc.data();
    TB_TRY((run_tiles<float, KT>(M, nd, nh, p, k, nodes, offsets, e, it.data(), nullptr, s, oc)));
    for (int c = 0; c < k; ++c) itot[(size_t)c] += it[(size_t)c];
    ppr_add_kernel<<<grid, 256, 0, s>>>(d_out, e, total);
    TB_CUDA(cudaGetLastError());
  }
  TB_CUDA(cudaStreamSynchronize(s));
  for (int c = 0; c < k; ++c) {
    if (iters_out) iters_out[c] = itot[(size_t)c];
    if (resid_out) resid_out[c] = res[(size_t)c];
  }
  return TBSLA_OK;
}

template <typename T>
tbsla_status_t run_kt(int kt, const tbsla_matrix *M, const int *nd, const std::vector<int> *nh,
                      const tbsla_pagerank_params_t *p, int k, const int *nodes, const int *offsets, double *out,
                      int *it, double *rs, cudaStream_t s) {
  switch (kt) {
  case 2: return run_tiles<T, 2>(M, nd, nh, p, k, nodes, offsets, out, it, rs, s);
  case 4: return run_tiles<T, 4>(M, nd, nh, p, k, nodes, offsets, out, it, rs, s);
  case 8: return run_tiles<T, 8>(M, nd, nh, p, k, nodes, offsets, out, it, rs, s);
  case 16: return run_tiles<T, 16>(M, nd, nh, p, k, nodes, offsets, out, it, rs, s);
  default: return run_tiles<T, 32>(M, nd, nh, p, k, nodes, offsets, out, it, rs, s);
  }
}

}  // namespace
}  // namespace tbsla

using namespace tbsla;

static tbsla_status_t ppr_batched(const tbsla_matrix_t *A, const tbsla_pagerank_params_t *p, int k,
                                  const int *nodes, const int *offsets, int tile, double *d_out, int *iterations,
                                  double *residuals, void *stream, bool refined) {
  TB_CHECK(A && p && nodes && offsets && d_out, "NULL argument");
  TB_CHECK(k > 0, "k = %d", k);
  TB_CHECK(A->format == TBSLA_FMT_CSR, "batched PageRank needs a CSR handle");
  TB_CHECK(A->n_row == A->n_col && A->rows == A->n_row && A->f_col == 0, "batched PageRank needs a square graph");
  TB_CHECK(p->precision == TBSLA_F64 || p->precision == TBSLA_F32, "precision must be TBSLA_F64 or TBSLA_F32");
  TB_CHECK(tile == 0 || tile == 2 || tile == 4 || tile == 8 || tile == 16 || tile == 32,
           "tile %d not 0, 2, 4, 8, 16 or 32", tile);
  TB_CUDA(cudaSetDevice(A->device));
  tbsla_matrix *M = const_cast<tbsla_matrix *>(A);
  tbsla_matrix *B = nullptr;
  TB_TRY(pr_relabelled(M, &B));
  const int *nd = B ? M->pr_newid : nullptr;
  const std::vector<int> *nh = B ? &M->pr_newid_host : nullptr;
  const tbsla_matrix *R = B ? B : M;
  const int tuned = M->ppr_tile[p->precision == TBSLA_F64 ? 0 : 1];
  // default: the widest tile the vectors fill (wide tiles stream the matrix
  // fewer times per vector: R-MAT 2^22, 256 vectors, FP64 ms per vector 15.8 /
  // 10.5 / 9.7 / 9.3 / 8.5 for tiles 2 / 4 / 8 / 16 / 32)
  const int kt = tile ? tile : tuned ? tuned : (k >= 32 ? 32 : k >= 16 ? 16 : k >= 8 ? 8 : k >= 4 ? 4 : 2);
  cudaStream_t s = (cudaStream_t)stream;
  if (refined) {
    TB_CHECK(p->precision == TBSLA_F32, "the refined batched solve takes TBSLA_F32");
    TB_CHECK(R->values[0] && R->values[1], "the refined batched solve needs the F64 and F32 value stores");
    switch (kt) {
    case 2: return run_refined<2>(R, nd, nh, p, k, nodes, offsets, d_out, iterations, residuals, s);
    case 4: return run_refined<4>(R, nd, nh, p, k, nodes, offsets, d_out, iterations, residuals, s);
    case 8: return run_refined<8>(R, nd, nh, p, k, nodes, offsets, d_out, iterations, residuals, s);
    case 16: return run_refined<16>(R, nd, nh, p, k, nodes, offsets, d_out, iterations, residuals, s);
    default: return run_refined<32>(R, nd, nh, p, k, nodes, offsets, d_out, iterations, residuals, s);
    }
  }
  if (p->precision == TBSLA_F64) return run_kt<double>(kt, R, nd, nh, p, k, nodes, offsets, d_out, iterations, residuals, s);
  return run_kt<float>(kt, R, nd, nh, p, k, nodes, offsets, d_out, iterations, residuals, s);
}

extern "C" tbsla_status_t tbsla_ppr_batched(const tbsla_matrix_t *A, const tbsla_pagerank_params_t *p, int k,
                                            const int *nodes, const int *offsets, int tile, double *d_out,
                                            int *iterations, double *residuals, void *stream) {
  return ppr_batched(A, p, k, nodes, offsets, tile, d_out, iterations, residuals, stream, false);
}

extern "C" tbsla_status_t tbsla_ppr_batched_refined(const tbsla_matrix_t *A, const tbsla_pagerank_params_t *p,
                                                    int k, const int *nodes, const int *offsets, int tile,
                                                    double *d_out, int *iterations, double *residuals,
                                                    void *stream) {
  return ppr_batched(A, p, k, nodes, offsets, tile, d_out, iterations, residuals, stream, true);
}
