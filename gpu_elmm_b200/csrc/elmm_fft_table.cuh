// elmm_fft_table.cuh -- the dispatch table of the register transforms.
#pragma once

#include "elmm_kernels.cuh"
#include "elmm_poisson_reg.cuh"

namespace elmm {

template <typename T, int N, bool INV>
constexpr auto ffty_reg_or_null() -> void (*)(const Dom<T> *, Launch, int) {
  if constexpr (fft_reg_y<T>(N)) return k_ffty_reg<T, N, INV>;
  else return nullptr;
}

template <typename T>
const FFTRegKernels<T> *fft_reg_kernels(int n) {
#define ELMM_REG_ENTRY(n_) \
  {n_, k_fftx_fwd_reg<T, n_>, k_fftx_inv_reg<T, n_>, ffty_reg_or_null<T, n_, false>(), ffty_reg_or_null<T, n_, true>()},
  static const FFTRegKernels<T> table[] = {ELMM_FFT_SIZES(ELMM_REG_ENTRY)};
#undef ELMM_REG_ENTRY
  for (const auto &e : table)
    if (e.n == n) return &e;
  return nullptr;
}

}  // namespace elmm
