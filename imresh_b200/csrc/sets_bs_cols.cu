// Column kernels of the Bluestein work lengths from 512.
#include "kernel_sets.cuh"

namespace imr {

template ColKernels col_set<-512>();
template ColKernels col_set<-1024>();
template ColKernels col_set<-2048>();
template ColKernels col_set<-4096>();

}  // namespace imr
