// The FP32-factor recompression kernel of single-system factorizations.
#include "blr_kernels.cuh"

namespace frank {
template __global__ void k_recompress<float>(BlrView<float>, FactorWs<float>, int, int, int, double, int, int*, int, double*, int*,
                                             int, int, int);
}  // namespace frank
