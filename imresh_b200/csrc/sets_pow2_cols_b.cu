// Column kernels of the power-of-two lengths from 1024.
#include "kernel_sets.cuh"

namespace imr {

template ColKernels col_set<1024>();
template ColKernels col_set<2048>();
template ColKernels col_set<4096>();

}  // namespace imr
