// elmm_fft_f64.cu -- the register transforms of every supported length in
// FP64 (elmm_poisson_reg.cuh), a translation unit of its own.
#include <cuda_runtime.h>

#include "elmm_fft_table.cuh"

namespace elmm {
template const FFTRegKernels<double> *fft_reg_kernels<double>(int n);
}  // namespace elmm
