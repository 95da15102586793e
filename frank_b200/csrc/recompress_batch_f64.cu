// The FP64 recompression kernel of batched factorizations.
#include "blr_kernels.cuh"

namespace frank {
template __global__ void k_recompress_b<double>(const SysDev<double>*, int);
}  // namespace frank
