// The FP32-factor recompression kernel of batched factorizations.
#include "blr_kernels.cuh"

namespace frank {
template __global__ void k_recompress_b<float>(const SysDev<float>*, int);
}  // namespace frank
