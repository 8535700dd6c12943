// elmm_fft_f32.cu -- the register transforms of every supported length in
// FP32 (elmm_poisson_reg.cuh), a translation unit of its own.
#include <cuda_runtime.h>

#include "elmm_fft_table.cuh"

namespace elmm {
template const FFTRegKernels<float> *fft_reg_kernels<float>(int n);
}  // namespace elmm
