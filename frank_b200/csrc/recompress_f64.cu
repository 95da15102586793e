// The FP64 recompression kernel of single-system factorizations.
#include "blr_kernels.cuh"

namespace frank {
template __global__ void k_recompress<double>(BlrView<double>, FactorWs<double>, int, int, int, double, int, int*, int, double*, int*,
                                             int, int, int);
}  // namespace frank
