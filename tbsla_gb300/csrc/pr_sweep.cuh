// pr_sweep.cuh -- the PageRank solver kernel: all sweeps of a solve in one
// cooperative launch.
//
// What bounds a solve: on graphs whose arrays fit in L2 not the bytes but the
// chain of dependent steps of one sweep (item -> column -> gathered value ->
// sum -> mass -> next term), and every kernel boundary in it adds a drain, a
// launch and a refill.  As one launch per row class, finalize, dot and
// combination (4 to 11 launches a sweep), the reference mode on cqmat 1e5 took
// 28 us a sweep and the accelerated adjoint on R-MAT 2^16 95 us; here a sweep
// is one pass over the row items, one grid barrier after which every block
// reduces the partial sums and advances the control block, and where the mode
// needs one an elementwise pass (Anderson combination) with its own barrier.
//
// Work split: one block of 1024 threads per SM (64 registers a thread), so that
// a barrier has few arrivals and few partial sums.  Rows are cut into classes
// so that a lane never walks more than a few batches of entries (solver_plan): 1,
// 4, 8 or 32 lanes a row, eight warps for a chunk of a longer row.  Each class is dealt round robin over all warps of
// the grid, beginning where the class before it ended.  A lane's entries go in
// batches whose index loads, then gathers, are in flight together.  The groups
// of a warp keep their sums until every lane holds a row, so the epilogue's
// FP64 instructions (2 lanes a clock and SM, the same cost with 1 or 32 lanes
// active) always serve 32 rows.
//
// Every block reduces the partial sums itself and advances its own copy of the
// control block (same inputs, same order, same bits), which saves the second
// hop of a barrier whose last arrival computes and releases; waiting blocks
// poll with relaxed loads (an acquire in the loop would drop the L1 lines of
// the warps still sweeping on the SM).
//
// Order: items, partial sums and chunk sums are added in fixed orders; results
// do not depend on scheduling.  The iterates are read with plain loads: they
// change during the launch (the barrier's fence drops the stale L1 lines),
// the matrix through the read-only path.
#pragma once

#include "anderson.cuh"
#include "csr_direct.cuh"

namespace tbsla {

// ------------------------------------------------------------ control
struct PrCtl {
  double beta, tol, inv_n, tele_scale;  // tele_scale: (1-beta)/n or (1-beta)/|P|
  double add;       // term of the next FP64 sweep (reference: tele; dangling: (b d + (1-b) s)/n)
  double add_in;    // term of the next inner sweep
  // reference mode: max of the new iterate; max of the iterate a sweep reads
  // (1: normalised); what its product is multiplied with; max of it over that of
  // the one before; the residual before `resid`
  double maxv, scale, beta_s, rho, resid_prev;
  int known, pass;  // resid is the read iterate's; the new iterate is normalised in place
  double resid, s;
  double inner_resid, inner_tol;
  double inner_eta; // inner tolerance relative to ||r||
  int iter, done, converged, max_iter;
  int inner_iter, inner_done, inner_max, inner_total;
  int f64_sweeps;
  int written;      // the result is in place
  // Anderson acceleration: for the last three sweep outputs (slot k % 3),
  // the sweep term each would give as the next input (linear in it), their
  // residuals' Gram matrix with the newest first (gram[i][j] = r_{k-i} .
  // r_{k-j}), and the coefficients of the next input in the newest-first
  // outputs.  aa: the FP64 solves; iaa: the inner (correction) solves of the
  // mixed-precision solve.
  struct Aa {
    double add[3];
    double gram[3][3];
    double coef[3];
    int m, pad;
  } aa, iaa;
};

enum { kSweepRef = 0, kSweepDang = 1, kSweepInner = 2, kSweepTele = 3, kSweepAdj = 4 };

// ------------------------------------------------------------ work list
// Classes: 0 chunks of eight warps, 1 / 2 / 3: 32 / 8 / 4 lanes, 4: one lane; of
// class 3 the last n_wide items take one lane that reads 16 bytes at a time
constexpr int kPrClasses = 5;
struct PrPlan {
  int4 *items = nullptr;       // (row, begin, end, chunk slot or -1), class by class
  int start[kPrClasses + 1] = {0, 0, 0, 0, 0, 0};
  int *empty = nullptr;        // rows without entries
  int n_empty = 0, n_wide = 0;
  int4 *chunks = nullptr;      // per chunk slot: (row, first slot of the row, chunks of the row, index of the row)
  int n_chunked = 0, slots = 0;
  int *arrived = nullptr;      // per chunked row: chunks summed so far (returns to 0 by itself)
  void *partial = nullptr;     // per chunk slot: its sum (8 bytes)
};

constexpr int kPrThreads = 1024;  // one block per SM
constexpr int kPrSub = 256;       // threads of one chunk
constexpr int kPrSubs = kPrThreads / kPrSub;

// What a sweep walks
enum { kPrItems = 0, kPrSlots = 1, kPrProduct = 2 };
template <typename V, typename T> struct PrMat {
  int layout;             // kPrItems: plan; kPrSlots: ELL layout; kPrProduct: prod holds A x
  PrPlan plan;
  const int *colidx;
  const V *values;
  const int *ecols;       // kPrSlots: slot j of row r at j * estride + r
  const V *evals;
  int64_t estride;
  int ewidth, rows, f_col;
  const T *prod;
};

// One launch of the solver
template <typename T> struct PrArgs {
  T *x[2];                // iterates: sweep k reads x[k & 1] (accelerated and mixed FP64: x[0])
  T *g[3], *r[3];         // accelerated: outputs and residuals, slot k % 3
  const unsigned char *dmask, *tmask;
  const double *tvec;     // teleport vector (adjoint: v, NULL uniform)
  const double *w;        // adjoint: right-hand side
  const float *rvec;      // inner: right-hand side
  double *x64;            // inner: the FP64 iterate the correction is added to
  float *r32, *e32;       // mixed: residual and first inner iterate
  double *out;            // result, in the labels of newid (NULL: none)
  const int *newid;
  double *partials;       // two buffers of 6 rows of part_stride doubles
  int part_stride;
  int n;
  int limit;              // sweeps of this launch at most
  int init;               // begin the solve: control block from ctl0, first iterate
  int mixed;              // this FP64 sweep serves the mixed-precision solve
  PrCtl *ctl;
  PrCtl ctl0;
  unsigned *bar;          // grid barrier: [0] arrivals of this launch, [kPrLeft] blocks that left, [kPrGaveUp]
  unsigned polls;         // of a barrier before a block gives up
};

// ------------------------------------------------------------ barrier
// All blocks of the (cooperative) grid meet: `target` is the arrival count
// that completes this barrier.  The wait is bounded by a number of polls (reads of
// L2, some tenths of a microsecond each), not by a clock: time while the context
// is off the GPU, which other contexts may share, is not counted.  A block
// that gives up raises bar[kPrGaveUp] for the host and kPrLost in the arrival
// count, and returns; every other block, whether it waits or arrives later and
// completes the count, sees the bit in the word it polls and returns too.
// (A launch has at most 10^6 sweeps of two barriers each on one block per SM: its
// arrivals stay far below that bit.)
constexpr int kPrLeft = 32, kPrGaveUp = 48, kPrBarWords = 64;  // words of the barrier, in lines of their own
constexpr unsigned kPrLost = 1u << 31;

__device__ __forceinline__ bool pr_barrier(unsigned *bar, unsigned &target, unsigned polls) {
  __shared__ int lost;
  target += gridDim.x;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(bar, 1u);
    unsigned seen = *(volatile unsigned *)bar;
    for (unsigned k = 0; seen < target; ++k) {  // kPrLost is above every target
      if (k >= polls) {
        atomicExch(bar + kPrGaveUp, 1u);
        seen = atomicOr(bar, kPrLost) | kPrLost;
        break;
      }
      seen = *(volatile unsigned *)bar;
    }
    lost = (seen & kPrLost) != 0;
    __threadfence();
  }
  __syncthreads();
  return !lost;
}

// ------------------------------------------------------------ reductions
// Per-thread values to partials[j * stride + slot], j < NV (sums; a maximum
// for j = 0 when take_max), three values at a time: eight warps per value add
// four threads' values each, one warp the rest, in a fixed order.
// sh: kPrShared doubles of shared memory.
constexpr int kPrShared = 3 * kPrThreads + 3 * 256;

// The maximum is taken by the order of the bits: fmax is several instructions of
// the FP64 pipe (reference mode on cqmat 1e5: this step 3.6 us, its reduction
// over the blocks 1.9 us; by bits 2.1 and 1.1).  Neither argument is a NaN.
__device__ __forceinline__ long long pr_key(double v) {
  const long long b = __double_as_longlong(v);
  return b ^ ((b >> 63) & 0x7fffffffffffffffLL);
}
__device__ __forceinline__ double pr_max(double a, double b) { return pr_key(a) < pr_key(b) ? b : a; }

template <int NV>
__device__ __forceinline__ void pr_block_partials(const double (&v)[NV], bool take_max, double *sh, double *partials,
                                                  int stride, int slot) {
  static_assert(kPrThreads == 1024, "eight warps of 128 threads' values for each value");
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  double *half = sh + 3 * kPrThreads;
  #pragma unroll
  for (int h = 0; h < NV; h += 3) {
    constexpr int M = 3;
    #pragma unroll
    for (int j = 0; j < M; ++j)
      if (h + j < NV) sh[j * kPrThreads + t] = v[h + j < NV ? h + j : 0];
    __syncthreads();
    if (warp < 8 * min(M, NV - h)) {
      const int j = warp >> 3;
      const bool mx = take_max && h + j == 0;
      const double *p = sh + j * kPrThreads + (warp & 7) * 128 + lane;
      const double a = mx ? pr_max(p[0], p[32]) : p[0] + p[32], b = mx ? pr_max(p[64], p[96]) : p[64] + p[96];
      half[j * 256 + (warp & 7) * 32 + lane] = mx ? pr_max(a, b) : a + b;
    }
    __syncthreads();
    if (warp < min(M, NV - h)) {
      const bool mx = take_max && h + warp == 0;
      double a = half[warp * 256 + lane];
      #pragma unroll
      for (int u = 1; u < 8; ++u) {
        const double b = half[warp * 256 + lane + 32 * u];
        a = mx ? pr_max(a, b) : a + b;
      }
      #pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const double b = __shfl_down_sync(0xffffffffu, a, o);
        a = mx ? pr_max(a, b) : a + b;
      }
      if (lane == 0) __stcg(partials + (size_t)(h + warp) * stride + slot, a);
    }
  }
}

// the partials [0, nparts) of every value, in a fixed order; valid in warp 0
template <int NV>
__device__ __forceinline__ void pr_reduce_partials(const double *partials, int stride, int nparts, bool take_max,
                                                   double (&v)[NV]) {
  __shared__ double sh[NV];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp < NV) {
    const bool mx = take_max && warp == 0;
    const double *p = partials + (size_t)warp * stride;
    double a = mx ? -INFINITY : 0.0;
    for (int k = lane; k < nparts; k += 256) {
      double b[8];
      #pragma unroll
      for (int u = 0; u < 8; ++u) b[u] = k + 32 * u < nparts ? __ldcg(p + k + 32 * u) : mx ? -INFINITY : 0.0;
      #pragma unroll
      for (int u = 0; u < 8; ++u) a = mx ? pr_max(a, b[u]) : a + b[u];
    }
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double b = __shfl_down_sync(0xffffffffu, a, o);
      a = mx ? pr_max(a, b) : a + b;
    }
    if (lane == 0) sh[warp] = a;
  }
  __syncthreads();
  if (warp == 0)
    #pragma unroll
    for (int j = 0; j < NV; ++j) v[j] = sh[j];
}

// The Anderson step after sweep k: the coefficients of the next input in the
// last three outputs (aa_coefficients).  They sum to 1, and the next sweep's
// term is affine in its input, so it is the same combination of the outputs'
// terms.
__device__ __forceinline__ double pr_anderson(PrCtl::Aa &st, int k, double term, double p0, double p1, double p2) {
  aa_gram_push(st.gram, p0, p1, p2);
  const int s0 = k % 3, s1 = (k + 2) % 3, s2 = (k + 1) % 3;  // slots of g_k, g_{k-1}, g_{k-2}
  st.add[s0] = term;
  st.m = aa_coefficients(st.gram, k < 2 ? k : 2, st.coef);
  double add = st.coef[0] * st.add[s0];
  if (st.m >= 1) add += st.coef[1] * st.add[s1];
  if (st.m >= 2) add += st.coef[2] * st.add[s2];
  return add;
}

// Reference mode, after sweep k: b = u / max(u) is left undone.  The update is
// linear in b up to its teleport term, itself a multiple of sum(b), so a sweep
// reads the unnormalised u_k, scales its product and term by the power of two
// that brings max(u_k) to [1, 2) (exact, where the division rounded every
// entry), and finds on the way what the sweep before it changed, u_k / max(u_k)
// - u_{k-1} / max(u_{k-1}): a sweep is one pass and one barrier.  With a pass
// of its own that divides (4.4 of 17 us a sweep on cqmat 1e5, and a barrier)
// 112 sweeps took 1888 us, now 1390 to 1440.  The convergence test comes one sweep
// late, and that sweep is lost when it says stop; so the pass that divides and
// tests at once runs where the test may hold (the last sweep allowed; the first
// two; the residual, should it go on falling as it did, below 1.25 tol), and
// where the maximum is no ordinary positive number (a negative one turns the vector
// round, which a power of two would not).  Runs in a warp, the two divisions in two
// lanes (each is a chain of some twenty FP64 instructions; five of them in
// one thread: 2.1 us a sweep).
__device__ __forceinline__ void pr_ref_advance(PrCtl &c, int k, double mx, double sum, double change) {
  const int lane = threadIdx.x & 31;
  const double q = lane ? change / c.scale : mx / c.scale;
  const double resid = __shfl_sync(0xffffffffu, q, 1);
  if (lane) return;
  c.maxv = mx;
  if (!c.known) {
    c.resid_prev = c.resid;
    c.resid = resid;
    if (c.resid < c.tol) {  // iterate k is the result; the new one is dropped
      c.converged = c.done = 1;
      return;
    }
  }
  c.iter = k + 1;
  c.f64_sweeps += 1;
  c.pass = k < 2 || c.iter >= c.max_iter || !(mx > 1e-30 && mx < 1e30) ||
           c.resid * (c.resid < c.resid_prev ? c.resid : c.resid_prev) < 1.25 * c.tol * c.resid_prev;
  if (!c.pass) {
    c.known = 0;
    c.scale = mx;
    c.rho = q;
    const double p = __longlong_as_double((2046ll << 52) - (__double_as_longlong(mx) & (2047ll << 52)));
    c.beta_s = c.beta * p;
    c.add = c.tele_scale * (sum * p);
  }
}

// ------------------------------------------------------------ epilogue
// A finished row: new value, and the thread's sums, in FP64 (the FP32 inner
// sweeps' change, which only stops the inner solve, in FP32; their mass and
// sum in pairs of FP32 numbers, six FP32 operations instead of a conversion
// and an FP64 addition): the maximum, the sum and the last sweep's change
// (reference); the change, the dangling mass (adjoint: v . lambda) and, where
// the next term needs it, the sum; accelerated, then the residual's dots with
// the last three residuals.
template <int MODE, typename T, bool AA> struct PrEmit {
  using Acc = T;
  static constexpr bool kSum = MODE == kSweepDang || MODE == kSweepInner;  // the sum is needed
  static constexpr int kBase = kSum || MODE == kSweepRef ? 3 : 2;
  static constexpr int NV = kBase + (AA ? 3 : 0);
  static constexpr bool kAccel = AA;
  T *y;
  const T *xold;
  T *r0;
  const T *r1, *r2;
  const unsigned char *dmask, *tmask;
  const double *tvec, *w;
  const float *rvec;
  double beta, add, inv_n, rho;
  int hist;  // accelerated: residuals stored before this sweep; reference: the last change is wanted
  T s0, s1, s2;
  double d0, d1, d2;
  float e1, e2;  // inner: the rounding errors of s1 and s2 (Knuth's two-sum)
  __device__ __forceinline__ static void two_sum(float &hi, float &lo, float v) {
    const float s = __fadd_rn(hi, v), t = __fsub_rn(s, hi);
    lo = __fadd_rn(lo, __fadd_rn(__fsub_rn(hi, __fsub_rn(s, t)), __fsub_rn(v, t)));
    hi = s;
  }
  __device__ __forceinline__ void clear() {
    s0 = MODE == kSweepRef ? (T)-INFINITY : (T)0;
    s1 = s2 = 0;
    d0 = d1 = d2 = 0;
    e1 = e2 = 0;
  }
  __device__ __forceinline__ void emit(int row, T v) {
    T val;
    if constexpr (MODE == kSweepInner) {
      // e' = beta * G~e + add + r in FP32
      val = __fmaf_rn((float)beta, (float)v, (float)add) + (float)rvec[row];
    } else if constexpr (MODE == kSweepRef) {
      val = __fma_rn(beta, v, tmask ? (tmask[row] ? add : 0.0) : add);
    } else if constexpr (MODE == kSweepDang) {
      val = __fma_rn(beta, v, add);
    } else if constexpr (MODE == kSweepTele) {
      val = __fma_rn(beta, v, add * tvec[row]);
    } else {
      // lambda' = beta A^T lambda + w + dangling * (beta v . lambda)
      val = __fma_rn(beta, v, w[row] + (dmask[row] ? add : 0.0));
    }
    if constexpr (MODE == kSweepRef) {
      // the change the last sweep made, up to its scale
      if (hist) s2 += fabs(fma(-rho, __ldcg(y + row), __ldcg(xold + row)));
      s0 = val > s0 ? val : s0;
      s1 += val;
    }
    __stcg(y + row, val);
    if constexpr (MODE != kSweepRef) {
      const T r = val - __ldcg(xold + row);
      s0 += MODE == kSweepInner ? (T)fabsf((float)r) : (T)fabs((double)r);
      if constexpr (MODE == kSweepAdj) {
        s1 += (tvec ? tvec[row] : inv_n) * val;
      } else {
        if constexpr (MODE == kSweepInner) {
          if (dmask[row]) two_sum(s1, e1, val);
          two_sum(s2, e2, val);
        } else {
          if (dmask[row]) s1 += val;
          if (kSum) s2 += val;
        }
      }
      if constexpr (AA) {
        __stcg(r0 + row, r);
        const double rd = (double)r;
        d0 += rd * rd;
        if (hist >= 1) d1 += rd * (double)__ldcg(r1 + row);
        if (hist >= 2) d2 += rd * (double)__ldcg(r2 + row);
      }
    }
  }
  __device__ __forceinline__ void sums(double (&v)[NV]) const {
    v[0] = (double)s0;
    if constexpr (kBase >= 2) v[1] = (double)s1 + (double)e1;
    if constexpr (kBase >= 3) v[2] = (double)s2 + (double)e2;
    if constexpr (AA) {
      v[kBase] = d0;
      v[kBase + 1] = d1;
      v[kBase + 2] = d2;
    }
  }
};

// ------------------------------------------------------------ sweep
// A batch: entries k, k + L, .., k + (U-1) L of a range that ends at b, their
// columns and values in flight together
template <typename V> struct PrBatch {
  static constexpr int U = 4;  // 8: no faster, FP32 registers spill
  int c[U];
  V v[U];
};
template <int L, typename V>
__device__ __forceinline__ void pr_load(PrBatch<V> &q, const int *__restrict__ colidx, const V *__restrict__ values,
                                        int k, int b) {
  #pragma unroll
  for (int u = 0; u < PrBatch<V>::U; ++u) {
    const bool in = k + u * L < b;
    q.c[u] = in ? ld_stream(colidx + k + u * L) : -1;
    q.v[u] = in ? ld_stream(values + k + u * L) : V(0);
  }
}
// its gathers, then one FMA per entry in order; `next` is loaded (nk, nb)
// between them, so that its latency overlaps the gathers'
template <int L, typename V, typename T>
__device__ __forceinline__ T pr_sum(T acc, PrBatch<V> &q, const PrMat<V, T> &m, const T *x, int nk, int nb) {
  T xv[PrBatch<V>::U];
  #pragma unroll
  for (int u = 0; u < PrBatch<V>::U; ++u) xv[u] = q.c[u] >= 0 ? x[q.c[u] - m.f_col] : T(0);
  PrBatch<V> next;
  pr_load<L, V>(next, m.colidx, m.values, nk, nb);
  #pragma unroll
  for (int u = 0; u < PrBatch<V>::U; ++u)
    if (q.c[u] >= 0) acc = fma_acc(to_acc(q.v[u], T()), xv[u], acc);
  q = next;
  return acc;
}

// Rows of one class, L lanes each, entries a + lane, a + lane + L, ... of a
// row to its lanes.  The next batch of entries (of this row or the warp's
// next) and the item after that are always in flight (asking L2 for entries
// further on gained nothing).  All lanes of a group end with the row's sum;
// round j of a warp leaves it to the lanes with lane % L == j % L, and after L
// rounds every lane emits a row of its own.
template <int L, typename V, typename T, typename E>
__device__ __forceinline__ void pr_sweep_groups(const PrMat<V, T> &m, const int4 *items, int n, int vw, int nw,
                                                const T *x, E &e) {
  constexpr int G = 32 / L;
  const int lane = threadIdx.x & 31, gl = lane & (L - 1), step = nw * G;
  const int4 none = make_int4(-1, 0, 0, -1);
  int base = vw * G;
  if (base >= n) return;
  int i = base + lane / L;
  int4 it = i < n ? __ldg(items + i) : none;
  i += step;
  int4 nx = i < n ? __ldg(items + i) : none;
  PrBatch<V> q;
  pr_load<L, V>(q, m.colidx, m.values, it.y + gl, it.z);
  int row = -1;
  T val = 0;
  for (int round = 0; base < n; base += step, ++round) {
    i += step;
    const int4 nn = i < n ? __ldg(items + i) : none;
    T s = 0;
    for (int k = it.y;;) {
      k += L * PrBatch<V>::U;
      const bool more = k < it.z;
      s = pr_sum<L, V, T>(s, q, m, x, (more ? k : nx.y) + gl, more ? it.z : nx.z);
      if (!more) break;
    }
    #pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (L == 1) {
      if (it.x >= 0) e.emit(it.x, s);
    } else {
      if ((round & (L - 1)) == gl) {
        row = it.x;
        val = s;
      }
      if ((round & (L - 1)) == L - 1) {
        if (row >= 0) e.emit(row, val);
        row = -1;
      }
    }
    it = nx;
    nx = nn;
  }
  if (L > 1 && row >= 0) e.emit(row, val);
}

// Four entries from a multiple of four, those outside [a, b) with column -1 (the
// arrays carry 64 bytes more than their entries)
__device__ __forceinline__ void pr_ld4(const double *p, double (&v)[4]) {
  const double2 a = __ldg(reinterpret_cast<const double2 *>(p)), b = __ldg(reinterpret_cast<const double2 *>(p + 2));
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void pr_ld4(const float *p, float (&v)[4]) {
  const float4 a = __ldg(reinterpret_cast<const float4 *>(p));
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
}
__device__ __forceinline__ void pr_ld4(const __nv_bfloat16 *p, __nv_bfloat16 (&v)[4]) {
  const uint2 a = __ldg(reinterpret_cast<const uint2 *>(p));
  v[0] = __ushort_as_bfloat16((unsigned short)a.x);
  v[1] = __ushort_as_bfloat16((unsigned short)(a.x >> 16));
  v[2] = __ushort_as_bfloat16((unsigned short)a.y);
  v[3] = __ushort_as_bfloat16((unsigned short)(a.y >> 16));
}
template <typename V>
__device__ __forceinline__ void pr_load4(PrBatch<V> &q, const int *__restrict__ colidx, const V *__restrict__ values,
                                         int k, int a, int b) {
  static_assert(PrBatch<V>::U == 4, "four entries");
  if (k < b) {
    pr_ld4(values + k, q.v);
    const int4 c = __ldg(reinterpret_cast<const int4 *>(colidx + k));
    q.c[0] = c.x; q.c[1] = c.y; q.c[2] = c.z; q.c[3] = c.w;
  }
  #pragma unroll
  for (int u = 0; u < 4; ++u)
    if (k + u < a || k + u >= b) q.c[u] = -1;
}

// Short rows, one lane each, four entries with 16-byte loads at a time through L1,
// which keeps the lines between the lanes of a warp.  FP32 and BF16 have the
// next four (of this row or the warp's next) in flight with the gathers; in
// FP64 and in accelerated FP32 sweeps their registers spill, the next row's
// bounds alone are (rules and times: solver_plan).
template <typename V, typename T, typename E>
__device__ __forceinline__ void pr_sweep_rows(const PrMat<V, T> &m, const int4 *items, int n, int vw, int nw,
                                              const T *x, E &e) {
  constexpr bool kAhead = sizeof(V) < (E::kAccel ? 4 : 8);
  const int lane = threadIdx.x & 31, step = nw * 32;
  const int4 none = make_int4(-1, 0, 0, -1);
  int i = vw * 32 + lane;
  int4 it = i < n ? __ldg(items + i) : none;
  i += step;
  int4 nx = i < n ? __ldg(items + i) : none;
  PrBatch<V> q;
  T xv[4];
  auto gather = [&]() {
    #pragma unroll
    for (int u = 0; u < 4; ++u) xv[u] = q.c[u] >= 0 ? x[q.c[u] - m.f_col] : T(0);
  };
  auto add = [&](T s) {
    #pragma unroll
    for (int u = 0; u < 4; ++u)
      if (q.c[u] >= 0) s = fma_acc(to_acc(q.v[u], T()), xv[u], s);
    return s;
  };
  if constexpr (kAhead) pr_load4<V>(q, m.colidx, m.values, it.y & ~3, it.y, it.z);
  for (int base = vw * 32; base < n; base += step) {
    T s = 0;
    if constexpr (kAhead) {
      i += step;
      const int4 nn = i < n ? __ldg(items + i) : none;
      for (int k = it.y & ~3;;) {
        k += 4;
        const bool more = k < it.z;
        gather();
        PrBatch<V> next;
        pr_load4<V>(next, m.colidx, m.values, more ? k : nx.y & ~3, more ? it.y : nx.y, more ? it.z : nx.z);
        s = add(s);
        q = next;
        if (!more) break;
      }
      if (it.x >= 0) e.emit(it.x, s);
      it = nx;
      nx = nn;
    } else {
      #pragma unroll 1
      for (int k = it.y & ~3; k < it.z; k += 4) {
        pr_load4<V>(q, m.colidx, m.values, k, it.y, it.z);
        gather();
        s = add(s);
      }
      if (it.x >= 0) e.emit(it.x, s);
      it = nx;
      i += step;
      nx = i < n ? __ldg(items + i) : none;
    }
  }
}

// One sweep over the block's share: sums of rows to e.emit, partial sums to
// the block's slot (chunked rows: to a slot per row after the blocks')
template <bool kWide, int MODE, typename V, typename T, bool AA>
__device__ __forceinline__ void pr_sweep(const PrMat<V, T> &m, const T *x, PrEmit<MODE, T, AA> &e, double *sh,
                                         double *partials, int stride) {
  constexpr int NV = PrEmit<MODE, T, AA>::NV;
  const int nb = gridDim.x, b = blockIdx.x;
  e.clear();
  if (kWide || m.layout == kPrItems) {
    const PrPlan &p = m.plan;
    // class 0: chunks, eight warps each.  The first warp of the eight adds the
    // threads' sums (in buffers used in turn, one barrier a chunk) and leaves
    // a finished row to lane (count % 32); 32 of them are emitted together.
    const int sub = threadIdx.x / kPrSub, st = threadIdx.x & (kPrSub - 1), cstep = nb * kPrSubs;
    T *part = reinterpret_cast<T *>(sh) + sub * 2 * kPrSub;
    const int4 none = make_int4(-1, 0, 0, -1);
    int ci = p.start[0] + sub * nb + b;
    if (ci < p.start[1]) {
      int4 it = __ldg(p.items + ci);
      PrBatch<V> q;
      pr_load<kPrSub, V>(q, m.colidx, m.values, it.y + st, it.z);
      int row = -1, count = 0;
      T val = 0;
      for (int buf = 0; ci < p.start[1]; buf ^= 1) {
        ci += cstep;
        const int4 nx = ci < p.start[1] ? __ldg(p.items + ci) : none;
        T acc = 0;
        for (int k = it.y;;) {
          k += kPrSub * PrBatch<V>::U;
          const bool more = k < it.z;
          acc = pr_sum<kPrSub, V, T>(acc, q, m, x, (more ? k : nx.y) + st, more ? it.z : nx.z);
          if (!more) break;
        }
        part[buf * kPrSub + st] = acc;
        asm volatile("bar.sync %0, %1;" ::"r"(1 + sub), "n"(kPrSub) : "memory");
        if (st < 32) {
          T s = part[buf * kPrSub + st];
          #pragma unroll
          for (int u = 1; u < kPrSub / 32; ++u) s += part[buf * kPrSub + st + 32 * u];
          #pragma unroll
          for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
          if (it.w < 0) {
            if (count == st) {
              row = it.x;
              val = s;
            }
            if (++count == 32) {
              e.emit(row, val);
              row = -1;
              count = 0;
            }
          } else if (st == 0) {
            // the chunk that arrives last adds the row's chunks in order; its
            // sums go to the row's own slot, so that they are the same
            // whichever block that is
            T *cp = static_cast<T *>(p.partial);
            const int4 ch = __ldg(p.chunks + it.w);  // row, first slot, chunks, index
            __stcg(cp + it.w, s);
            __threadfence();
            if (atomicInc((unsigned *)p.arrived + ch.w, (unsigned)ch.z - 1) == (unsigned)ch.z - 1) {
              __threadfence();
              T t = 0;
              for (int c0 = 0; c0 < ch.z; c0 += 8) {
                T u[8];
                #pragma unroll
                for (int c = 0; c < 8; ++c) u[c] = c0 + c < ch.z ? __ldcg(cp + ch.y + c0 + c) : T(0);
                #pragma unroll
                for (int c = 0; c < 8; ++c) t += u[c];
              }
              PrEmit<MODE, T, AA> er = e;
              er.clear();
              er.emit(ch.x, t);
              double v[NV];
              er.sums(v);
              #pragma unroll
              for (int j = 0; j < NV; ++j) __stcg(partials + (size_t)j * stride + nb + ch.w, v[j]);
            }
          }
          __syncwarp();
        }
        it = nx;
      }
      if (st < 32 && row >= 0) e.emit(row, val);
    }
    // warp w of the grid lies in block w % nb: small classes spread over all SMs
    const int nw = nb * (kPrThreads / 32), w = (threadIdx.x >> 5) * nb + b;
    const int n32 = p.start[2] - p.start[1], n8 = p.start[3] - p.start[2], n4 = p.start[4] - p.start[3] - (kWide ? p.n_wide : 0),
              n1 = p.start[5] - p.start[4];
    int off = (p.start[1] - p.start[0]) * (kPrSub / 32) % nw;
    auto begin = [&](int units) {  // this class's first warp is the one after the last class's last
      int vw = w - off;
      if (vw < 0) vw += nw;
      off = (off + units) % nw;
      return vw;
    };
    if (n32) pr_sweep_groups<32, V, T>(m, p.items + p.start[1], n32, begin(n32), nw, x, e);
    if (n8) pr_sweep_groups<8, V, T>(m, p.items + p.start[2], n8, begin((n8 + 3) / 4), nw, x, e);
    if (n4) pr_sweep_groups<4, V, T>(m, p.items + p.start[3], n4, begin((n4 + 7) / 8), nw, x, e);
    if constexpr (kWide)
      pr_sweep_rows<V, T>(m, p.items + p.start[4] - p.n_wide, p.n_wide, begin((p.n_wide + 31) / 32), nw, x, e);
    if (n1) pr_sweep_groups<1, V, T>(m, p.items + p.start[4], n1, begin((n1 + 31) / 32), nw, x, e);
    const int lane = threadIdx.x & 31;
    for (int i = begin(0) * 32 + lane; i < p.n_empty; i += nw * 32) e.emit(__ldg(p.empty + i), T(0));
  } else if (m.layout == kPrSlots) {
    // ELL layout: one lane per row, coalesced, eight slots in flight; padding
    // of the CSR handles' copy holds column -1, an ELL handle's column below
    // f_col reads x[0] (MatrixELL.cpp:108-109)
    for (int r = b * kPrThreads + threadIdx.x; r < m.rows; r += nb * kPrThreads) {
      T acc = 0;
      for (int j0 = 0; j0 < m.ewidth; j0 += 8) {
        int c[8];
        V v[8];
        T xv[8];
        #pragma unroll
        for (int u = 0; u < 8; ++u) {
          const bool in = j0 + u < m.ewidth;
          c[u] = in ? ld_ell<false>(m.ecols + (size_t)(j0 + u) * m.estride + r) : -1;
          v[u] = in ? ld_ell<false>(m.evals + (size_t)(j0 + u) * m.estride + r) : V(0);
        }
        #pragma unroll
        for (int u = 0; u < 8; ++u) xv[u] = c[u] >= 0 ? x[max(c[u] - m.f_col, 0)] : T(0);
        #pragma unroll
        for (int u = 0; u < 8; ++u)
          if (c[u] >= 0) acc = fma_acc(to_acc(v[u], T()), xv[u], acc);
      }
      e.emit(r, acc);
    }
  } else {
    for (int r = b * kPrThreads + threadIdx.x; r < m.rows; r += nb * kPrThreads) e.emit(r, m.prod[r]);
  }
  double v[NV];
  e.sums(v);
  __syncthreads();  // the chunks' use of sh
  pr_block_partials<NV>(v, MODE == kSweepRef, sh, partials, stride, b);
}

// ------------------------------------------------------------ the solver
// MODE kSweepInner: T = float, the correction solve of the mixed-precision
// solve; otherwise T = V = double.  kWide: row items with wide ones among them, in
// a kernel of its own, since the registers of one walk cost the others (both in
// one: R-MAT 2^23 adjoint 17.5 ms, 16.1 without).  The arguments of a launch are best
// left in their places: four bytes more in front of the pointers of PrMat, and every
// sweep of the 4-lane class took a tenth longer.
template <bool kWide, int MODE, typename V, typename T, bool AA>
__global__ void __launch_bounds__(kPrThreads, 1) pr_solve_kernel(const PrMat<V, T> m, const PrArgs<T> a) {
  constexpr bool kInner = MODE == kSweepInner;
  constexpr int NV = PrEmit<MODE, T, AA>::NV, NB = PrEmit<MODE, T, AA>::kBase;
  __shared__ double sh[kPrShared];
  __shared__ PrCtl c;  // every block's copy; block 0 stores it at the end
  const int nb = gridDim.x, b = blockIdx.x, n = a.n;
  const int t0 = b * kPrThreads + threadIdx.x, nt = nb * kPrThreads;
  unsigned target = 0, phase = 0;
  const int st = a.part_stride;
  auto buffer = [&]() { return a.partials + (size_t)(phase & 1) * 6 * st; };
  // the end of a phase: the blocks meet, and the first `lanes` threads advance
  // the control block from the reduced sums
  auto meet = [&](auto values, int nparts, bool take_max, auto advance, int lanes = 1) {
    constexpr int N = sizeof(values) / sizeof(double);
    if (!pr_barrier(a.bar, target, a.polls)) return false;
    double u[N];
    pr_reduce_partials<N>(buffer(), st, nparts, take_max, u);
    ++phase;
    if (threadIdx.x < lanes) advance(u);
    __syncthreads();
    return true;
  };
  struct V1 { double v[1]; };
  struct V2 { double v[2]; };
  struct VN { double v[NV]; };
  if (!kInner && a.init) {
    // first iterate: reference 1 (0.25 with nodes), dangling 1/n, teleport v,
    // adjoint w; its mass gives the first sweep's term
    if (threadIdx.x == 0) {
      c = a.ctl0;
      c.scale = 1.0;
      c.beta_s = c.beta;
      c.known = 1;
    }
    double v[2] = {0, 0};  // dangling mass (adjoint: v . w), sum
    for (int i = t0; i < n; i += nt) {
      double x0;
      if constexpr (MODE == kSweepRef) x0 = a.tmask ? 0.25 : 1.0;
      else if constexpr (MODE == kSweepDang) x0 = a.ctl0.inv_n;
      else if constexpr (MODE == kSweepTele) x0 = a.tvec[i];
      else if constexpr (MODE == kSweepAdj) x0 = a.w[i];
      else x0 = 0;
      __stcg(a.x[0] + i, (T)x0);
      if constexpr (MODE == kSweepAdj) {
        v[0] += (a.tvec ? a.tvec[i] : a.ctl0.inv_n) * x0;
      } else {
        if (MODE != kSweepRef && a.dmask[i]) v[0] += x0;
        v[1] += x0;
      }
    }
    pr_block_partials<2>(v, false, sh, buffer(), st, b);
    if (!meet(V2{}, nb, false, [&](const double (&u)[2]) {
          if constexpr (MODE == kSweepRef) c.add = c.tele_scale * u[1];
          else if constexpr (MODE == kSweepDang) c.add = (c.beta * u[0] + (1.0 - c.beta) * u[1]) * c.inv_n;
          else if constexpr (MODE == kSweepTele) c.add = c.beta * u[0] + (1.0 - c.beta);
          else c.add = c.beta * u[0];
        }))
      return;
  } else {
    for (int w = threadIdx.x; w < (int)(sizeof(PrCtl) / 8); w += kPrThreads)
      reinterpret_cast<double *>(&c)[w] = __ldcg(reinterpret_cast<const double *>(a.ctl) + w);
    __syncthreads();
  }
  const bool skip = kInner && (c.done || c.inner_done);
  for (int step = 0; !skip && step < a.limit; ++step) {
    if (kInner ? c.inner_done : c.done) break;
    const int k = kInner ? c.inner_iter : c.iter;
    const int s0 = k % 3, s1 = (k + 2) % 3, s2 = (k + 1) % 3;
    PrEmit<MODE, T, AA> e;
    const T *x = AA || a.mixed ? a.x[0] : a.x[k & 1];
    e.y = AA ? a.g[s0] : a.mixed ? a.x[1] : a.x[(k + 1) & 1];
    e.xold = x;
    e.r0 = AA ? a.r[s0] : nullptr;
    e.r1 = AA ? a.r[s1] : nullptr;
    e.r2 = AA ? a.r[s2] : nullptr;
    e.dmask = a.dmask;
    e.tmask = a.tmask;
    e.tvec = a.tvec;
    e.w = a.w;
    e.rvec = a.rvec;
    e.beta = MODE == kSweepRef ? c.beta_s : c.beta;
    e.rho = c.rho;
    e.add = kInner ? c.add_in : c.add;
    e.inv_n = c.inv_n;
    e.hist = MODE == kSweepRef ? !c.known : k;
    T *const yk = e.y;
    pr_sweep<kWide, MODE, V, T, AA>(m, x, e, sh, buffer(), st);
    const int nparts = nb + (m.layout == kPrItems ? m.plan.n_chunked : 0);
    if (!meet(VN{}, nparts, MODE == kSweepRef, [&](const double (&v)[NV]) {
          if constexpr (MODE == kSweepRef) {
            pr_ref_advance(c, k, v[0], v[1], v[2]);
          } else if constexpr (kInner) {
            const double term = (c.beta * v[1] + (1.0 - c.beta) * v[2]) * c.inv_n;
            c.inner_resid = v[0];
            c.inner_iter = k + 1;
            c.inner_done = v[0] < c.inner_tol || c.inner_iter >= c.inner_max;
            if constexpr (AA) c.add_in = pr_anderson(c.iaa, k, term, v[NB], v[NB + 1], v[NB + 2]);
            else c.add_in = term;
          } else {
            double term;
            if constexpr (MODE == kSweepDang) term = (c.beta * v[1] + (1.0 - c.beta) * v[2]) * c.inv_n;
            else if constexpr (MODE == kSweepTele) term = c.beta * v[1] + (1.0 - c.beta);
            else term = c.beta * v[1];
            c.resid = v[0];
            c.iter = k + 1;
            c.f64_sweeps += 1;
            c.converged = v[0] < c.tol;
            c.done = c.converged || c.iter >= c.max_iter;
            if constexpr (AA) c.add = pr_anderson(c.aa, k, term, v[NB], v[NB + 1], v[NB + 2]);
            else c.add = term;
          }
        }, MODE == kSweepRef ? 32 : 1))
      return;
    if constexpr (MODE == kSweepRef) {
      if (c.done) break;
      if (c.pass) {
        // b /= max; sums of |b - b_prev| and of b
        double v[2] = {0, 0};
        const double mx = c.maxv, sc = c.scale;
        for (int i = t0; i < n; i += nt) {
          const double q = __ldcg(yk + i) / mx, p = __ldcg(x + i);
          __stcg(yk + i, (T)q);
          v[0] += fabs(q - (sc == 1.0 ? p : p / sc));
          v[1] += q;
        }
        pr_block_partials<2>(v, false, sh, buffer(), st, b);
        if (!meet(V2{}, nb, false, [&](const double (&u)[2]) {
              c.resid_prev = c.resid;
              c.resid = u[0];
              c.known = 1;
              c.scale = 1.0;
              c.beta_s = c.beta;
              c.add = c.tele_scale * u[1];
              c.converged = u[0] < c.tol;
              c.done = c.converged || c.iter >= c.max_iter;
            }))
          return;
      }
    }
    if constexpr (AA) {
      if (!(kInner ? c.inner_done : c.done)) {
        // x_{k+1} = c0 g_k + c1 g_{k-1} + c2 g_{k-2} (only the terms in use are read)
        const PrCtl::Aa &aa = kInner ? c.iaa : c.aa;
        const T c0 = (T)aa.coef[0], c1 = (T)aa.coef[1], c2 = (T)aa.coef[2];
        const int mm = aa.m;
        for (int i = t0; i < n; i += nt) {
          T q = c0 * __ldcg(a.g[s0] + i);
          if (mm >= 1) q = fma(c1, __ldcg(a.g[s1] + i), q);
          if (mm >= 2) q = fma(c2, __ldcg(a.g[s2] + i), q);
          __stcg(a.x[0] + i, q);
        }
        if (!pr_barrier(a.bar, target, a.polls)) return;
      }
    }
  }
  if constexpr (kInner) {
    if (!skip && c.inner_done) {
      // x += e, and the mass of the corrected x for the next FP64 sweep
      const int k = c.inner_iter;
      const T *el = AA ? a.g[(k + 2) % 3] : a.x[k & 1];
      double v[2] = {0, 0};
      for (int i = t0; i < n; i += nt) {
        const double q = __ldcg(a.x64 + i) + (double)__ldcg(el + i);
        __stcg(a.x64 + i, q);
        if (a.dmask[i]) v[0] += q;
        v[1] += q;
      }
      pr_block_partials<2>(v, false, sh, buffer(), st, b);
      if (!meet(V2{}, nb, false, [&](const double (&u)[2]) {
            c.add = (c.beta * u[0] + (1.0 - c.beta) * u[1]) * c.inv_n;
            c.inner_total += c.inner_iter;
          }))
        return;
    }
  } else if (a.mixed && !c.done) {
    if (a.limit > 0) {
      // r = x1 - x0 in FP32, e0 = r, and the mass of e0
      double v[2] = {0, 0};
      for (int i = t0; i < n; i += nt) {
        const float d = (float)(__ldcg(a.x[1] + i) - __ldcg(a.x[0] + i));
        a.r32[i] = d;
        a.e32[i] = d;
        if (a.dmask[i]) v[0] += (double)d;
        v[1] += (double)d;
      }
      pr_block_partials<2>(v, false, sh, buffer(), st, b);
      if (!meet(V2{}, nb, false, [&](const double (&u)[2]) {
            c.add_in = (c.beta * u[0] + (1.0 - c.beta) * u[1]) * c.inv_n;
            c.inner_iter = 0;
            c.inner_done = 0;
            c.inner_tol = c.inner_eta * c.resid;
          }))
        return;
    }
  } else if (c.done && !c.written) {
    // the result; reference and mixed: b /= sum(b) (Matrix.cpp:52-59)
    const int k = c.iter;
    const T *xr = k == 0 ? a.x[0] : a.mixed ? a.x[1] : AA ? a.g[(k + 2) % 3] : a.x[k & 1];
    if (MODE == kSweepRef || a.mixed) {
      double v[1] = {0};
      for (int i = t0; i < n; i += nt) v[0] += (double)__ldcg(xr + i);
      pr_block_partials<1>(v, false, sh, buffer(), st, b);
      if (!meet(V1{}, nb, false, [&](const double (&u)[1]) { c.s = u[0]; })) return;
      const double s = c.s;
      for (int i = t0; i < n; i += nt) a.out[i] = __ldcg(xr + (a.newid ? a.newid[i] : i)) / s;
    } else {
      for (int i = t0; i < n; i += nt) a.out[i] = __ldcg(xr + (a.newid ? a.newid[i] : i));
    }
    __syncthreads();
    if (threadIdx.x == 0) c.written = 1;
  }
  __syncthreads();
  if (b == 0)
    for (int w = threadIdx.x; w < (int)(sizeof(PrCtl) / 8); w += kPrThreads)
      reinterpret_cast<double *>(a.ctl)[w] = reinterpret_cast<const double *>(&c)[w];
  // the block that leaves last clears the barrier for the next launch
  if (threadIdx.x == 0 && atomicInc(a.bar + kPrLeft, gridDim.x - 1) == gridDim.x - 1) a.bar[0] = 0;
}

}  // namespace tbsla
