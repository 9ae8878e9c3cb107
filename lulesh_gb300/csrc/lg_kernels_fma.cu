// lg_kernels_fma.cu -- build of the cycle kernels in 64-bit fixed point, with FP64 (and
// FMA contraction) where values do not fit.
#define LG_NS fp64_fma
#define LG_NS_NAME "fp64_fma"
#define LG_REASSOC 1
#define LG_FIXED_EOS 1
#include "lg_kernels.cuh"
#include "lg_kernelset.inc"
namespace lg {
const KernelSet *kernels_fp64_fma() { return &fp64_fma::kKernelSet; }
}
