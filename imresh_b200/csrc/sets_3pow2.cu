// Kernels of the lengths 3 * 2^k.
#include "kernel_sets.cuh"

namespace imr {

template RowKernels row_set<192>();
template ColKernels col_set<192>();
template RowKernels row_set<384>();
template ColKernels col_set<384>();
template RowKernels row_set<768>();
template ColKernels col_set<768>();
template RowKernels row_set<1536>();
template ColKernels col_set<1536>();
template RowKernels row_set<3072>();
template ColKernels col_set<3072>();

}  // namespace imr
