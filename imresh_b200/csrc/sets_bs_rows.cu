// Row kernels of the Bluestein work lengths from 512.
#include "kernel_sets.cuh"

namespace imr {

template RowKernels row_set<-512>();
template RowKernels row_set<-1024>();
template RowKernels row_set<-2048>();
template RowKernels row_set<-4096>();

}  // namespace imr
