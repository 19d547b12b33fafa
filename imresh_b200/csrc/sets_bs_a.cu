// Kernels of the Bluestein work lengths up to 256.
#include "kernel_sets.cuh"

namespace imr {

template RowKernels row_set<-8>();
template ColKernels col_set<-8>();
template RowKernels row_set<-16>();
template ColKernels col_set<-16>();
template RowKernels row_set<-32>();
template ColKernels col_set<-32>();
template RowKernels row_set<-64>();
template ColKernels col_set<-64>();
template RowKernels row_set<-128>();
template ColKernels col_set<-128>();
template RowKernels row_set<-256>();
template ColKernels col_set<-256>();

}  // namespace imr
