// Column kernels of the power-of-two lengths up to 512.
#include "kernel_sets.cuh"

namespace imr {

template ColKernels col_set<64>();
template ColKernels col_set<128>();
template ColKernels col_set<256>();
template ColKernels col_set<512>();

}  // namespace imr
