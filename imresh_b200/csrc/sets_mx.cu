// Grouped-pass kernels of the lengths without a compile-time kernel.
#include "kernel_sets.cuh"

namespace imr {

RowKernels row_set_mx(int n)
{
    RowKernels k{k_row_hio_mx<true, false>, k_row_hio_mx<false, false>, k_row_finish_mx<0>, k_fft_rows_mx<-1>,
                 k_fft_rows_mx<+1>, std::max(1, kMxRowElems / n), kMxRowThreads, 0, nullptr, nullptr, 0, 0};
    k.smem = mx_row_smem(n, k.nb);
    k.hio_fix = k_row_hio_mx<false, true>;
    k.mx = 1;
    return k;
}
template <int T, int C>
static ColKernels col_set_mx_t(int n)
{
    ColKernels k{k_col_mx<0, T, C>, k_col_mx<1, T, C>, k_fft_cols_mx<-1, T, C>, k_fft_cols_mx<+1, T, C>, C, T,
                 mx_col_smem<C>(n), nullptr, 0, 0, 0, 0, 0};
    k.checks = 1;
    return k;
}
ColKernels col_set_mx(int n, int W)
{
    if (mx_few_columns(n, W)) return col_set_mx_t<512, kMxColWFew>(n);
    return mx_col_threads(n) == 256 ? col_set_mx_t<256, kMxColW>(n) : col_set_mx_t<512, kMxColW>(n);
}

}  // namespace imr
