// Per-length instantiation of the row/column pass kernels and their launchers.
// FP32 (tc == 0): the register-handoff kernels of cdx_rfft.cuh.  Tensor-core
// radix-16 passes: the staged kernels of cdx_kernels.cuh, on tcgen05 (tc == 1)
// or on warp-level mma.sync (tc == 2).
#pragma once
#include <atomic>

#include "cdx_rfft.cuh"

namespace cdx {

template <int N, int TCM>
cudaError_t prepare_tc_mode() {
  using G = Geom<N>;
  constexpr int X = TCM == 2 ? umma_smem_extra<N>() : 0;
  cudaError_t e;
  if ((e = cudaFuncSetAttribute(row_pass_kernel<N, ROW_FFT, TCM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                G::SMEM_LINES + X)) != cudaSuccess)
    return e;
  if ((e = cudaFuncSetAttribute(row_pass_kernel<N, ROW_ITER, TCM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                G::SMEM_ROW_ITER + X)) != cudaSuccess)
    return e;
  if ((e = cudaFuncSetAttribute(col_pass_kernel<N, COL_FFT, TCM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                G::SMEM_LINES + X)) != cudaSuccess)
    return e;
  // at 4096 the noise-tolerant projection's three staged tiles and the tcgen05
  // operands exceed a CTA's 227 KB: that one combination is refused at launch
  constexpr int CI = G::SMEM_COL_CCD + X <= 232448 ? G::SMEM_COL_CCD + X : G::SMEM_COL_ITER + X;
  return cudaFuncSetAttribute(col_pass_kernel<N, COL_ITER, TCM>, cudaFuncAttributeMaxDynamicSharedMemorySize, CI);
}

template <int N>
cudaError_t prepare_tc() {
  cudaError_t e = prepare_tc_mode<N, 1>();
  return e != cudaSuccess ? e : prepare_tc_mode<N, 2>();
}

template <class K>
cudaError_t max_smem(K* kernel, int bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}
template <class G, bool SQ>
cudaError_t prepare_row_g() {
  constexpr int SM = RGeom<G>::SMEM_ROW_ITER;
  cudaError_t e;
  if ((e = max_smem(row_pass_rk<G, ROW_ITER, ALGO_HIO, SQ>, SM)) != cudaSuccess) return e;
  if ((e = max_smem(row_pass_rk<G, ROW_ITER, ALGO_RAAR, SQ>, SM)) != cudaSuccess) return e;
  if ((e = max_smem(row_pass_rk<G, ROW_ITER, ALGO_ER, SQ>, SM)) != cudaSuccess) return e;
  if ((e = max_smem(row_pass_rk<G, ROW_ITER, ALGO_POSER, SQ>, SM)) != cudaSuccess) return e;
  if ((e = max_smem(row_pass_rk<G, ROW_ITER, ALGO_POSHIO, SQ>, SM)) != cudaSuccess) return e;
  return max_smem(row_pass_rk<G, ROW_ITER, ALGO_FHIO, SQ>, SM);
}
template <class G>
cudaError_t prepare_g() {
  cudaError_t e;
  if ((e = max_smem(row_pass_rk<G, ROW_FFT, ALGO_ER>, RGeom<G>::SMEM_ROW_LINES)) != cudaSuccess) return e;
  if ((e = prepare_row_g<G, false>()) != cudaSuccess) return e;
  if constexpr (row_sq_ok_g<G>()) if ((e = prepare_row_g<G, true>()) != cudaSuccess) return e;
  if ((e = max_smem(col_pass_rk<G, COL_FFT, PROJ_MODABS>, G::SMEM_LINES)) != cudaSuccess) return e;
  if ((e = max_smem(col_pass_rk<G, COL_ITER, PROJ_MODABS>, G::SMEM_COL_ITER)) != cudaSuccess) return e;
  return max_smem(col_pass_rk<G, COL_ITER, PROJ_CCD>, G::SMEM_COL_CCD);
}

template <int N>
cudaError_t prepare_rk() {
  using G = FGeom<N>;
  using W = WideGeom<N>;
  cudaError_t e = prepare_g<G>();
  if constexpr (ThinGeom<N>::T != G::T) if (e == cudaSuccess) e = prepare_g<ThinGeom<N>>();
  if constexpr (W::L != G::L)
    if (e == cudaSuccess) e = max_smem(col_pass_rk<W, COL_FFT, PROJ_MODABS, G::LOG2L>, W::SMEM_LINES);
  return e;
}

// Raise the dynamic shared-memory limit of the kernels of length N on the
// current device (outside any stream capture), once per device: the ~30 attribute
// calls of a length cost a transform's caller more than its two launches (96 x 192
// fields, a forward and an inverse transform: 54 -> 33 us).
template <int N>
cudaError_t prepare_len() {
  static std::atomic<unsigned long long> done{0};   // bit per device
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
  if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
  if ((e = prepare_rk<N>()) != cudaSuccess || (e = prepare_tc<N>()) != cudaSuccess) return e;
  done.fetch_or(bit, std::memory_order_release);
  return cudaSuccess;
}

// Programmatic dependent launch per length: measured on one GB300 it saves
// 1-2 % per iteration at 256^2 x64, 384^2 x16, 512^2 x16 and 1024^2 x4 and
// costs 1.3 % at 2048^2 (60.7 against 59.9 us), so that length launches plainly.
template <int N>
constexpr bool pass_pdl() { return N != 2048; }
// launch mode of a pass: the per-length default, or the autotuner's choice (1 plain, 2 PDL)
template <int N>
bool pdl_of(int mode) { return mode == 0 ? pass_pdl<N>() : mode == 2; }

template <class G>
cudaError_t launch_row_g(const RowArgs& a, int batch, cudaStream_t st) {
  constexpr int N = G::N, SM = RGeom<G>::SMEM_ROW_ITER;
  const dim3 grid((a.rows + G::L - 1) / G::L, batch);
  const bool pdl = pdl_of<N>(a.pdl_mode);
  if (a.mode != ROW_ITER)
    return launch_pdl(row_pass_rk<G, ROW_FFT, ALGO_ER>, grid, G::T, RGeom<G>::SMEM_ROW_LINES, st, a, pdl);
  if constexpr (row_sq_ok_g<G>()) if (row_sq_layout<G>(a)) switch (a.algo) {   // the compile-time layout of square patterns
    case ALGO_HIO: return launch_pdl(row_pass_rk<G, ROW_ITER, ALGO_HIO, true>, grid, G::T, SM, st, a, pdl);
    case ALGO_RAAR: return launch_pdl(row_pass_rk<G, ROW_ITER, ALGO_RAAR, true>, grid, G::T, SM, st, a, pdl);
    case ALGO_ER: return launch_pdl(row_pass_rk<G, ROW_ITER, ALGO_ER, true>, grid, G::T, SM, st, a, pdl);
    case ALGO_POSER: return launch_pdl(row_pass_rk<G, ROW_ITER, ALGO_POSER, true>, grid, G::T, SM, st, a, pdl);
    case ALGO_POSHIO: return launch_pdl(row_pass_rk<G, ROW_ITER, ALGO_POSHIO, true>, grid, G::T, SM, st, a, pdl);
    default: return launch_pdl(row_pass_rk<G, ROW_ITER, ALGO_FHIO, true>, grid, G::T, SM, st, a, pdl);
  }
  switch (a.algo) {   // unknown codes take the FHIO branch, as applySupport does (cdi.cc:25-36)
    case ALGO_HIO: return launch_pdl(row_pass_rk<G, ROW_ITER, ALGO_HIO>, grid, G::T, SM, st, a, pdl);
    case ALGO_RAAR: return launch_pdl(row_pass_rk<G, ROW_ITER, ALGO_RAAR>, grid, G::T, SM, st, a, pdl);
    case ALGO_ER: return launch_pdl(row_pass_rk<G, ROW_ITER, ALGO_ER>, grid, G::T, SM, st, a, pdl);
    case ALGO_POSER: return launch_pdl(row_pass_rk<G, ROW_ITER, ALGO_POSER>, grid, G::T, SM, st, a, pdl);
    case ALGO_POSHIO: return launch_pdl(row_pass_rk<G, ROW_ITER, ALGO_POSHIO>, grid, G::T, SM, st, a, pdl);
    default: return launch_pdl(row_pass_rk<G, ROW_ITER, ALGO_FHIO>, grid, G::T, SM, st, a, pdl);
  }
}

template <int N>
cudaError_t launch_row(const RowArgs& a, int batch, cudaStream_t st) {
  using G = Geom<N>;
  dim3 grid((a.rows + G::L - 1) / G::L, batch);
  if (a.tc == 1) {   // tcgen05 (the kernels' TCM 2)
    constexpr int X = umma_smem_extra<N>();
    if (a.mode == ROW_ITER) row_pass_kernel<N, ROW_ITER, 2><<<grid, G::T, G::SMEM_ROW_ITER + X, st>>>(a);
    else row_pass_kernel<N, ROW_FFT, 2><<<grid, G::T, G::SMEM_LINES + X, st>>>(a);
  } else if (a.tc == 2) {   // mma.sync (the kernels' TCM 1)
    if (a.mode == ROW_ITER) row_pass_kernel<N, ROW_ITER, 1><<<grid, G::T, G::SMEM_ROW_ITER, st>>>(a);
    else row_pass_kernel<N, ROW_FFT, 1><<<grid, G::T, G::SMEM_LINES, st>>>(a);
  } else {
    if constexpr (ThinGeom<N>::T != FGeom<N>::T) if (a.thin) return launch_row_g<ThinGeom<N>>(a, batch, st);
    return launch_row_g<FGeom<N>>(a, batch, st);
  }
  return cudaGetLastError();
}

template <class G>
cudaError_t launch_col_g(const ColArgs& a, int batch, cudaStream_t st) {
  const dim3 grid((a.cols + G::L - 1) / G::L, batch);
  const bool pdl = pdl_of<G::N>(a.pdl_mode);
  if (a.mode != COL_ITER) return launch_pdl(col_pass_rk<G, COL_FFT, PROJ_MODABS>, grid, G::T, G::SMEM_LINES, st, a, pdl);
  if (a.proj == PROJ_CCD) return launch_pdl(col_pass_rk<G, COL_ITER, PROJ_CCD>, grid, G::T, G::SMEM_COL_CCD, st, a, pdl);
  return launch_pdl(col_pass_rk<G, COL_ITER, PROJ_MODABS>, grid, G::T, G::SMEM_COL_ITER, st, a, pdl);
}

template <int N>
cudaError_t launch_col(const ColArgs& a, int batch, cudaStream_t st) {
  using G = Geom<N>;
  dim3 grid((a.cols + G::L - 1) / G::L, batch);
  const int smem_iter = a.proj == PROJ_CCD ? G::SMEM_COL_CCD : G::SMEM_COL_ITER;
  if (a.tc == 1) {
    constexpr int X = umma_smem_extra<N>();
    if (a.mode == COL_ITER) col_pass_kernel<N, COL_ITER, 2><<<grid, G::T, smem_iter + X, st>>>(a);
    else col_pass_kernel<N, COL_FFT, 2><<<grid, G::T, G::SMEM_LINES + X, st>>>(a);
  } else if (a.tc == 2) {
    if (a.mode == COL_ITER) col_pass_kernel<N, COL_ITER, 1><<<grid, G::T, smem_iter, st>>>(a);
    else col_pass_kernel<N, COL_FFT, 1><<<grid, G::T, G::SMEM_LINES, st>>>(a);
  } else {
    using F = FGeom<N>;
    if constexpr (ThinGeom<N>::T != F::T) if (a.thin) return launch_col_g<ThinGeom<N>>(a, batch, st);
    if constexpr (WideGeom<N>::L != F::L) {
      // row-major output, and enough columns to give every SM a wide CTA
      using W = WideGeom<N>;
      const int w = (a.cols + W::L - 1) / W::L;
      if (a.mode != COL_ITER && !a.out_tiled && (long long)w * batch >= sm_count())
        return launch_pdl(col_pass_rk<W, COL_FFT, PROJ_MODABS, F::LOG2L>, dim3(w, batch), W::T, W::SMEM_LINES, st, a,
                          pdl_of<N>(a.pdl_mode));
    }
    return launch_col_g<F>(a, batch, st);
  }
  return cudaGetLastError();
}

#define CDX_INSTANTIATE(N)                                                   \
  template cudaError_t prepare_len<N>();                                     \
  template cudaError_t launch_row<N>(const RowArgs&, int, cudaStream_t);     \
  template cudaError_t launch_col<N>(const ColArgs&, int, cudaStream_t);

}  // namespace cdx
