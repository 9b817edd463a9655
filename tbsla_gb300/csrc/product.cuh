// product.cuh -- launches of the SpMV kernels of every format with an
// epilogue functor (plain products, a_axpx).
//
// Every epilogue provides emit(row, v), which receives each finished row
// exactly once.
#pragma once

#include <algorithm>

#include "common.cuh"
#include "csr_direct.cuh"
#include "csr_rows.cuh"
#include "spmv_kernels.cuh"

namespace tbsla {

// grids: one row (one row item) per thread (group), the most loads in flight;
// the staged kernel strides a grid of at most kStrideBlocks blocks
constexpr int kStrideBlocks = 152 * 16;
inline int short_grid(int64_t n_short) { return (int)std::max<int64_t>(1, (n_short + 255) / 256); }
inline int group_grid(int n_items, int lanes) {
  const int per_block = 256 / lanes;
  return (int)std::max<int64_t>(1, ((int64_t)n_items + per_block - 1) / per_block);
}
inline int fixup_grid(int n) { return std::max(1, (n + 127) / 128); }

template <typename Acc> inline Carry<Acc> carry_of(const tbsla_matrix *A);
template <> inline Carry<double> carry_of<double>(const tbsla_matrix *A) {
  return Carry<double>{A->tile_head_row, A->tile_head_val, A->tile_tail_val, A->tile_emitted};
}
template <> inline Carry<float> carry_of<float>(const tbsla_matrix *A) {
  return Carry<float>{A->tile_head_row, A->tile_head_val32, A->tile_tail_val32, A->tile_emitted};
}

// ------------------------------------------------------------ launches
// Dynamic shared memory of csr_rows_kernel (set once per instantiation).
template <typename V, typename XT, typename Epi> size_t csr_rows_setup() {
  constexpr size_t smem = csr_rows_smem<typename Epi::Acc>();
  static bool done = false;
  if (!done) {
    cudaFuncSetAttribute(csr_rows_kernel<V, XT, Epi>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    done = true;
  }
  return smem;
}

template <typename Acc> inline Acc *huge_partials_of(const tbsla_matrix *A);
template <> inline double *huge_partials_of<double>(const tbsla_matrix *A) { return A->huge_partials; }
template <> inline float *huge_partials_of<float>(const tbsla_matrix *A) { return A->huge_partials32; }
template <typename Acc> inline Acc *chunk_partials_of(const tbsla_matrix *A);
template <> inline double *chunk_partials_of<double>(const tbsla_matrix *A) { return A->chunk_partials; }
template <> inline float *chunk_partials_of<float>(const tbsla_matrix *A) { return A->chunk_partials32; }

// The handle's L2 policy on the gathered vector (x of type XT).  The range
// form needs the vector's bytes in 32 bits; larger vectors keep a fraction.
template <typename XT> inline XKeep xkeep_of(const tbsla_matrix *A) {
  XKeep k{A->x_keep, 0u};
  const int64_t bytes = A->x_extent * (int64_t)sizeof(XT);
  if (A->x_keep_range && bytes > 0 && bytes <= (int64_t)0xffffffffll) k.range = (uint32_t)bytes;
  return k;
}

// The staged kernel applies when every row is short (stage_cap > 0) and the
// handle's stage mode (tbsla_matrix_tune) is on.
inline bool stage_on(const tbsla_matrix *A) {
  return A->stage_cap > 0 && A->short_rows == nullptr && A->short_mode == 1 &&
         A->stage_cap <= kStageCapMax;
}
// dynamic shared memory of csr_stage_kernel (the attribute is raised once per
// instantiation to the largest capacity)
template <typename V, typename XT, typename Epi> size_t csr_stage_setup(int cap) {
  static bool done = false;
  if (!done) {
    cudaFuncSetAttribute(csr_stage_kernel<V, XT, Epi>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)csr_stage_smem<V>(kStageCapMax));
    done = true;
  }
  return csr_stage_smem<V>(cap);
}

// Rows per thread of csr_sell_kernel: the handle's setting, else 2 (cqmat
// 7e4 to 1.6e7 rows, c 8 to 32, FP32 and FP64: 2 the fastest or within 3 %;
// the 2^24 FP64 product 0.625 ms against 0.646 with 4 and more with 1)
inline int sell_rows_per_thread(const tbsla_matrix *A) {
  return A->sell_rows > 0 ? A->sell_rows : 2;
}

// The sliced copy of the value store `vals` (csr_sell_kernel), when the
// handle has one and plain products take it: the default short-row mode, or
// mode 3; F64 and F32 stores (BF16 slots load 64 bytes per warp instruction:
// cqmat 2^24 0.366 ms against 0.334 with one thread per row)
template <typename V> inline const V *sell_vals_for(const tbsla_matrix *A, const V *vals) {
  if constexpr (sizeof(V) < 4) {
    return nullptr;  // BF16: the copy is not kept
  } else {
    if (!A->sell_width || !(A->short_mode == -1 || A->short_mode == 3)) return nullptr;
    for (int k = 0; k < 2; ++k)
      if (A->values[k] == static_cast<const void *>(vals)) return static_cast<const V *>(A->sell_vals[k]);
    return nullptr;
  }
}

// The direct CSR launches (row bins of the handle) over rowptr / colidx:
// the CSR arrays of a CSR handle, or the derived row pointer of a row-sorted
// COO handle.
template <typename V, typename XT, typename Epi>
tbsla_status_t launch_csr_direct(const tbsla_matrix *A, const int *rowptr, const int *colidx, const V *vals,
                                 const XT *x, Epi epi, cudaStream_t s) {
  using Acc = typename Epi::Acc;
  KernelTimer kt(A, s);
  if (const V *sv = sell_vals_for<V>(A, vals)) {
    // every row short, the ELL-layout copy: one warp per 32 R rows
    const int R = sell_rows_per_thread(A);
    const int64_t threads = A->sell_stride / (32 * R) * 32;
    const int grid = (int)((threads + 255) / 256);
    if (R == 4)
      csr_sell_kernel<4, V, XT, Epi><<<grid, 256, 0, s>>>(A->sell_cols, sv, A->sell_stride, A->sell_width, x,
                                                          A->f_col, A->rows, xkeep_of<XT>(A), epi);
    else if (R == 2)
      csr_sell_kernel<2, V, XT, Epi><<<grid, 256, 0, s>>>(A->sell_cols, sv, A->sell_stride, A->sell_width, x,
                                                          A->f_col, A->rows, xkeep_of<XT>(A), epi);
    else
      csr_sell_kernel<1, V, XT, Epi><<<grid, 256, 0, s>>>(A->sell_cols, sv, A->sell_stride, A->sell_width, x,
                                                          A->f_col, A->rows, xkeep_of<XT>(A), epi);
    kt.stop();
    return TBSLA_OK;
  }
  // two lanes per short row: asked for, or FP64 values and rows long enough
  const bool pair = A->short_mode == 2 || (A->short_mode < 0 && sizeof(V) == 8 &&
                                           A->short_nnz >= (int64_t)kPairMinRow * A->n_short);
  if (A->n_short > 0 && stage_on(A)) {
    // all rows short: the staged kernel
    const size_t smem = csr_stage_setup<V, XT, Epi>(A->stage_cap);
    const int tiles = (A->n_short + 31) / 32;
    const int grid = std::max(1, std::min((tiles + kStageWarps - 1) / kStageWarps, kStrideBlocks));
    csr_stage_kernel<V, XT, Epi><<<grid, kStageWarps * 32, smem, s>>>(A->n_short, rowptr, colidx, vals, x, A->f_col,
                                                                     xkeep_of<XT>(A), A->stage_cap, epi);
  } else if (A->n_short > 0 && A->short_rows == nullptr && A->short_mode < 0 && A->short_max <= kTinyRow) {
    // every row in order and tiny: warp tiles of 32 * 8 / T rows
    const int T = A->short_max <= 2 ? 2 : 4;
    const int64_t warps = ((int64_t)A->n_short + 32 * (8 / T) - 1) / (32 * (8 / T));
    const int grid = (int)((warps * 32 + 255) / 256);
    if (T == 2)
      csr_tiny_kernel<2, V, XT, Epi><<<grid, 256, 0, s>>>(A->n_short, rowptr, colidx, vals, x, A->f_col,
                                                          xkeep_of<XT>(A), epi);
    else
      csr_tiny_kernel<4, V, XT, Epi><<<grid, 256, 0, s>>>(A->n_short, rowptr, colidx, vals, x, A->f_col,
                                                          xkeep_of<XT>(A), epi);
  } else if (A->n_warp_items == 0 && A->n_short > 0 && pair) {
    csr_pair_kernel<V, XT, Epi><<<short_grid(2 * (int64_t)A->n_short), 256, 0, s>>>(
        A->n_short, rowptr, colidx, vals, x, A->f_col, xkeep_of<XT>(A), epi);
  } else if (A->n_warp_items == 0 && A->n_short > 0) {
    csr_short_kernel<V, XT, Epi><<<short_grid(A->n_short), 256, 0, s>>>(A->n_short, rowptr, colidx, vals, x, A->f_col,
                                                                       xkeep_of<XT>(A), epi);
  } else if (A->n_warp_items > 0) {
    // long rows: every class and the short rows in one launch
    MixedPlan p{};
    p.items = A->warp_items;
    p.rows = A->short_rows;
    p.n_short = A->n_short;
    for (int c = 0; c <= kGroupClasses; ++c) p.start[c] = A->item_class_start[c];
    int blocks = 0;
    for (int c = kGroupClasses - 1; c >= 0; --c) {
      p.first[c] = blocks;
      const int n = p.start[c + 1] - p.start[c];
      if (n > 0) blocks += group_grid(n, kGroupLanes[c]);
    }
    p.first[kGroupClasses] = blocks;
    Acc *parts = chunk_partials_of<Acc>(A);
    if (A->n_short > 0) blocks += short_grid((pair ? 2 : 1) * (int64_t)A->n_short);
    const bool plain = sizeof(V) >= 4 && p.start[3] - p.start[2] >= kPlainItems;
    auto launch = [&](auto kernel) {
      kernel<<<blocks, 256, 0, s>>>(p, rowptr, colidx, vals, x, A->f_col, xkeep_of<XT>(A), parts, epi);
    };
    if (pair) launch(plain ? csr_mixed_kernel<true, true, V, XT, Epi> : csr_mixed_kernel<true, false, V, XT, Epi>);
    else launch(plain ? csr_mixed_kernel<false, true, V, XT, Epi> : csr_mixed_kernel<false, false, V, XT, Epi>);
  }
  kt.stop();
  if (A->n_chunk_rows > 0) {
    csr_chunk_fixup_kernel<Epi><<<fixup_grid(A->n_chunk_rows), 128, 0, s>>>(
        A->chunk_rows, A->n_chunk_rows, chunk_partials_of<Acc>(A), epi);
  }
  return TBSLA_OK;
}

// DENSE products by dense_rows_kernel: few columns, and for FP32 and BF16 64 rows an
// SM (16 warps of four; with fewer the batches and splits of dense_kernel fill
// the GPU as well or better: 5000 x 256 FP32 5.5 us, here 6.8).  FP32 and BF16 up
// to 192 columns (10000 rows: 128 columns 5.9 us by dense_kernel, 5.4 here; 400 6.7 and
// 7.7), from 16384 rows 320 (20000 x 256 7.9, 6.9; 384 9.0, 9.8), from 32768,
// whose matrix leaves L2, 512 in FP32 (65536 rows 30.4, 26.5) and 400 in BF16 (384:
// 17.0, 13.7); BF16 whose rows do not start on 16 bytes up to 2048 (20000 x 1500
// 21.0, 16.0).  FP64, whose pipe is the bound, counts steps of 32 columns here and
// pairs of them there, and loses occupancy to dense_kernel's registers: up to 192
// columns (1500 x 128 7.9, 7.0; 256 7.3, 8.6), from 64 rows an SM 288 (20000 x 257
// 25.6, 23.9; 10000 x 512 19.8, 21.5), from 32768 rows always (33554 x 1000 89.7,
// 79.3; 20000 x 1500 70.5, 75.3), but not where the last, partial step is one of
// few (335544 x 100 180, 232).
template <typename V> inline bool dense_by_rows(int rows, int cols, bool vec) {
  if (sizeof(V) == 8) {
    if (cols % 32 != 0 && cols < 128 && 2 * ((cols + 63) / 64) == (cols + 31) / 32) return false;
    return cols <= (rows < 64 * 152 ? 192 : 288) || rows >= 32768;
  }
  if (rows < 64 * 152) return false;
  if (sizeof(V) == 2 && !vec) return cols <= 2048;
  return cols <= (rows >= 32768 ? (sizeof(V) == 4 ? 512 : 400) : rows >= 16384 ? 320 : 192);
}

template <typename V, typename XT, typename Epi>
tbsla_status_t launch_product(const tbsla_matrix *A, const V *vals, const XT *x, Epi epi,
                              cudaStream_t s) {
  using Acc = typename Epi::Acc;
  switch (A->format) {
  case TBSLA_FMT_CSR:
    if (A->rows > 0 && A->csr_variant == 0) {
      TB_TRY(launch_csr_direct<V, XT>(A, A->idx0, A->idx1, vals, x, epi, s));
    } else if (A->rows > 0) {
      const size_t smem = csr_rows_setup<V, XT, Epi>();
      KernelTimer kt(A, s);
      csr_rows_kernel<V, XT, Epi><<<A->num_blocks, kRowsNT, smem, s>>>(
          A->row_blocks, A->idx0, A->idx1, vals, x, A->f_col, huge_partials_of<Acc>(A), epi);
      kt.stop();
      if (A->num_huge > 0)
        csr_huge_fixup_kernel<Epi><<<(A->num_huge + 127) / 128, 128, 0, s>>>(A->huge_rows, A->num_huge,
                                                                            huge_partials_of<Acc>(A), epi);
    }
    break;
  case TBSLA_FMT_COO:
  case TBSLA_FMT_SCOO:
    if (A->stored > 0 && A->coo_rowptr && A->csr_variant == 0) {
      TB_TRY(launch_csr_direct<V, XT>(A, A->coo_rowptr, A->idx1, vals, x, epi, s));
    } else if (A->stored > 0) {
      KernelTimer kt(A, s);
      coo_merge_kernel<kMergeThreads, kMergeItems, V, XT, Epi><<<A->num_tiles, kMergeThreads, 0, s>>>(
          A->idx0, A->idx1, vals, x, A->f_col, A->stored, carry_of<Acc>(A), epi);
      kt.stop();
      merge_fixup_kernel<Epi><<<(A->num_tiles + 255) / 256, 256, 0, s>>>(A->num_tiles, carry_of<Acc>(A), epi);
    }
    break;
  case TBSLA_FMT_ELL:
    if (A->rows > 0 && A->max_col > 0) {
      const bool cs = A->x_extent * (int64_t)sizeof(XT) <= (64ll << 20);
      KernelTimer kt(A, s);
      if (A->csr_variant == 0) {
        // warp tiles of 32 R rows (the default), R rows per thread
        // (TBSLA_TUNE_SELL_ROWS)
        const int R = sell_rows_per_thread(A);
        const int64_t threads = ((int64_t)A->rows + 32 * R - 1) / (32 * R) * 32;
        const int grid = (int)((threads + 255) / 256);
        const XKeep k = xkeep_of<XT>(A);
        if (cs && R == 4)
          ell_warp_kernel<V, XT, Epi, true, 4><<<grid, 256, 0, s>>>(A->idx0, vals, x, A->f_col, A->rows,
                                                                    A->rows_pad, A->max_col, k, epi);
        else if (cs && R == 2)
          ell_warp_kernel<V, XT, Epi, true, 2><<<grid, 256, 0, s>>>(A->idx0, vals, x, A->f_col, A->rows,
                                                                    A->rows_pad, A->max_col, k, epi);
        else if (cs)
          ell_warp_kernel<V, XT, Epi, true, 1><<<grid, 256, 0, s>>>(A->idx0, vals, x, A->f_col, A->rows,
                                                                    A->rows_pad, A->max_col, k, epi);
        else if (R == 4)
          ell_warp_kernel<V, XT, Epi, false, 4><<<grid, 256, 0, s>>>(A->idx0, vals, x, A->f_col, A->rows,
                                                                     A->rows_pad, A->max_col, k, epi);
        else if (R == 2)
          ell_warp_kernel<V, XT, Epi, false, 2><<<grid, 256, 0, s>>>(A->idx0, vals, x, A->f_col, A->rows,
                                                                     A->rows_pad, A->max_col, k, epi);
        else
          ell_warp_kernel<V, XT, Epi, false, 1><<<grid, 256, 0, s>>>(A->idx0, vals, x, A->f_col, A->rows,
                                                                     A->rows_pad, A->max_col, k, epi);
      } else {
        // four consecutive rows per thread
        const int threads = (A->rows + 3) / 4;
        if (cs)
          ell_kernel<V, XT, Epi, true><<<(threads + 255) / 256, 256, 0, s>>>(A->idx0, vals, x, A->f_col, A->rows,
                                                                             A->rows_pad, A->max_col, xkeep_of<XT>(A), epi);
        else
          ell_kernel<V, XT, Epi, false><<<(threads + 255) / 256, 256, 0, s>>>(A->idx0, vals, x, A->f_col, A->rows,
                                                                              A->rows_pad, A->max_col, xkeep_of<XT>(A), epi);
      }
      kt.stop();
    }
    break;
  case TBSLA_FMT_DENSE:
    if (A->rows > 0 && A->cols > 0) {
      // 16-byte loads when every row and x start on 16 bytes
      constexpr int VW = 16 / (int)sizeof(V);
      const bool vec = A->cols % VW == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
      KernelTimer kt(A, s);
      if (dense_by_rows<V>(A->rows, A->cols, vec)) {
        dense_rows_kernel<V, XT, Epi><<<(int)(((int64_t)A->rows + 31) / 32), 256, 0, s>>>(vals, x, A->rows, A->cols, epi);
        kt.stop();
        break;
      }
      // warps per row group: as many as leave each four steps of columns, so
      // that blocks are short and many (8000 x 9001 FP64 in blocks of 35 steps,
      // one wave and a tenth: 281 us, against 175 with few, long blocks)
      const int64_t groups = ((int64_t)A->rows + dense_rows<V>() - 1) / dense_rows<V>();
      const int batch = 32 * (vec ? VW * dense_steps<V, VW>() : dense_steps<V, 1>());  // columns of a warp's step
      int splits = 1;
      while (splits < 8 && A->cols / (2 * splits) >= 4 * batch) splits *= 2;
      while (splits < 8 && groups * splits < 152 * 6 && A->cols / (2 * splits) >= 128) splits *= 2;
      const int grid = (int)((groups * splits + 7) / 8);
      if (vec) dense_kernel<VW, V, XT, Epi><<<grid, 256, 0, s>>>(vals, x, A->rows, A->cols, splits, epi);
      else dense_kernel<1, V, XT, Epi><<<grid, 256, 0, s>>>(vals, x, A->rows, A->cols, splits, epi);
      kt.stop();
    }
    break;
  default:
    return fail(TBSLA_ERR_INVALID_ARG, "unknown format %d", A->format);
  }
  TB_CUDA(cudaGetLastError());
  return TBSLA_OK;
}

}  // namespace tbsla
