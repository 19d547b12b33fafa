// Row kernels of the power-of-two lengths.
#include "kernel_sets.cuh"

namespace imr {

template RowKernels row_set<64>();
template RowKernels row_set<128>();
template RowKernels row_set<256>();
template RowKernels row_set<512>();
template RowKernels row_set<1024>();
template RowKernels row_set<2048>();
template RowKernels row_set<4096>();

}  // namespace imr
