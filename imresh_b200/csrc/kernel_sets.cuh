// The kernels and launch shapes of each compile-time length and Bluestein work
// length (N < 0: work length -N).  Instantiated by the sets_*.cu files, one
// class of lengths each, so that the classes compile in parallel.
#pragma once
#include <algorithm>

#include "engine_host.hpp"
#include "kernels.cuh"

namespace imr {

template <int N>
static void add_shapes(RowKernels &k)
{
    if constexpr (narrow_length(N)) {
        k.n_hio_first = k_row_hio_n<true, N>;
        k.n_hio = k_row_hio_n<false, N>;
        k.n_hio_fix = k_row_hio_n<false, N, true>;
        k.n_nb = row_n_rows(N);
        k.n_threads = row_n_threads(N);
        k.n_smem = row_n_smem(N);
    }
}
template <int N>
static void add_shapes(ColKernels &k)
{
    if constexpr (is_pow2(N) && fcol_narrow(N)) {
        k.f_fwd = k_fft_cols_r<-1, N, kFcolN>;
        k.f_inv = k_fft_cols_r<+1, N, kFcolN>;
        k.f_nb = kFcolN;
        k.f_threads = kFcolN * N / 8;
        k.f_smem = reg_smem_bytes(N, kFcolN);
    }
    if constexpr (narrow_length(N)) {
        k.n_col = k_col_n<N>;
        k.n_nb = kColN;
        k.n_threads = col_n_threads(N);
        k.n_smem = col_n_smem(N);
    }
}

template <int N>
RowKernels row_set()
{
    RowKernels k{};
    if constexpr (N >= 16 && is_pow2(N)) {
        k = RowKernels{k_row_hio_r<true, N>, k_row_hio_r<false, N>, k_row_finish_r<N>,
                       k_fft_rows_r<-1, N>, k_fft_rows_r<+1, N>, rrow_nb(N), rrow_threads(N),
                       rrow_smem(N), k_row_hio_p<true, N>, k_row_hio_p<false, N>,
                       prow_smem<true, N>(), prow_smem<false, N>()};
        k.hio_fix = k_row_hio_r<false, N, true>;
        k.p_hio_fix = k_row_hio_p<false, N, true>;
        k.p_finish = k_row_finish_p<N>;
        k.p_smem_fin = pfin_smem<N>();
        add_shapes<N>(k);
    } else if constexpr (N >= 8 && is_pow2(N)) {
        k = RowKernels{k_row_hio_r<true, N>, k_row_hio_r<false, N>, k_row_finish_r<N>,
                       k_fft_rows_r<-1, N>, k_fft_rows_r<+1, N>, rrow_nb(N), rrow_threads(N),
                       rrow_smem(N), nullptr, nullptr, 0, 0};
        k.hio_fix = k_row_hio_r<false, N, true>;
    } else if constexpr (is_3pow2(N)) {   // per-tile kernels + pipelined 12-value register passes
        k = RowKernels{k_row_hio<true, N>, k_row_hio<false, N>, k_row_finish<N>, k_fft_rows<-1, N>,
                       k_fft_rows<+1, N>, row_nb(N), row_threads(N), 0, k_row_hio_p<true, N>,
                       k_row_hio_p<false, N>, prow_smem<true, N>(), prow_smem<false, N>()};
        k.hio_fix = k_row_hio<false, N, true>;
        k.p_hio_fix = k_row_hio_p<false, N, true>;
        k.p_finish = k_row_finish_p<N>;
        k.p_smem_fin = pfin_smem<N>();
        add_shapes<N>(k);
    } else if constexpr (N < 0 && -N >= 256) {   // Bluestein lengths, 16 values per thread
        constexpr int M = -N;
        k = RowKernels{k_row_hio_bs16<true, M>, k_row_hio_bs16<false, M>, k_row_finish_bs16<M>,
                       k_fft_rows_bs16<-1, M>, k_fft_rows_bs16<+1, M>, bs16_rows(M), bs16_row_threads(M),
                       bs16_row_smem(M), nullptr, nullptr, 0, 0};
        k.hio_fix = k_row_hio_bs16<false, M, true>;
    } else if constexpr (N < 0 && -N >= 8) {   // Bluestein lengths: register chirp-z transforms
        constexpr int M = -N;
        k = RowKernels{k_row_hio_bs<true, M>, k_row_hio_bs<false, M>, k_row_finish_bs<M>, k_fft_rows_bs<-1, M>,
                       k_fft_rows_bs<+1, M>, rrow_nb(M), rrow_threads(M), rrow_smem(M), nullptr, nullptr, 0, 0};
        k.hio_fix = k_row_hio_bs<false, M, true>;
    } else {
        static_assert(N >= 8 && is_pow2(N), "no kernels for this length class");
    }
    return k;
}
template <int N>
ColKernels col_set()
{
    if constexpr (N >= 128 && N <= 4096 && is_pow2(N)) {   // 16 values per thread in the pipelined pass
        constexpr int T = pcol16_nbt(N);
        ColKernels k{k_col_r<N>, k_col_init_r<N>, k_fft_cols_r<-1, N, rcol_nb(N)>, k_fft_cols_r<+1, N, rcol_nb(N)>,
                     rcol_nb(N), rcol_threads(N), rcol_smem(N), k_col_p16<N, T, false>, pcol16_smem<N, T>(),
                     pcol_box_rows(N), 0, pcol16_threads(N, T), T, 1};
        if constexpr (N >= 256) {   // split-precision tensor-core variants
            k.p_col_tc[0] = k_col_tc<N, T, kPrecBf16x3, 0>;
            k.p_col_tc[1] = k_col_tc<N, T, kPrecFp16x3, 0>;
            k.fft_tc[0][0] = k_col_tc<N, T, kPrecBf16x3, 1>;
            k.fft_tc[0][1] = k_col_tc<N, T, kPrecBf16x3, 2>;
            k.fft_tc[1][0] = k_col_tc<N, T, kPrecFp16x3, 1>;
            k.fft_tc[1][1] = k_col_tc<N, T, kPrecFp16x3, 2>;
            k.p_smem_tc = pcol_tc_smem<N, T>();
        }
        add_shapes<N>(k);
        if constexpr (T >= 4) k.p_col_split = k_col_p16<N, T, true>;   // half tiles of >= 2 columns (16-byte TMA rows)
        return k;
    } else if constexpr (N >= 16 && is_pow2(N)) {
        ColKernels k{k_col_r<N>, k_col_init_r<N>, k_fft_cols_r<-1, N, rcol_nb(N)>, k_fft_cols_r<+1, N, rcol_nb(N)>,
                     rcol_nb(N), rcol_threads(N), rcol_smem(N), k_col_p<N>, pcol_smem<N>(),
                     pcol_box_rows(N), pcol_tma_m(N) ? 1 : 0, pcol_threads(N), rcol_nb(N)};
        add_shapes<N>(k);
        return k;
    } else if constexpr (N >= 8 && is_pow2(N))
        return ColKernels{k_col_r<N>, k_col_init_r<N>, k_fft_cols_r<-1, N, rcol_nb(N)>, k_fft_cols_r<+1, N, rcol_nb(N)>,
                          rcol_nb(N), rcol_threads(N), rcol_smem(N), nullptr, 0, 0, 0, 0};
    else if constexpr (is_3pow2(N)) {
        ColKernels k{k_col<N>, k_col_init<N>, k_fft_cols<-1, N>, k_fft_cols<+1, N>, col_nb(N),
                     col_threads(N), 0, k_col_p<N>, pcol_smem<N>(), pcol_box_rows(N),
                     pcol_tma_m(N) ? 1 : 0, pcol_threads(N), rcol_nb(N)};
        add_shapes<N>(k);
        return k;
    } else if constexpr (N < 0 && -N >= 256)   // Bluestein lengths, 16 values per thread
    {
        ColKernels k{k_col_bs16<-N, 0>, k_col_bs16<-N, 1>, k_fft_cols_bs16<-1, -N>, k_fft_cols_bs16<+1, -N>,
                     bs16_col_nb(-N), bs16_col_threads(-N), bs16_col_smem(-N), nullptr, 0, 0, 0, 0, 0};
        k.checks = 1;
        return k;
    }
    else if constexpr (N < 0 && -N >= 8)   // Bluestein lengths: register chirp-z transforms
        return ColKernels{k_col_bs<-N>, k_col_init_bs<-N>, k_fft_cols_bs<-1, -N>, k_fft_cols_bs<+1, -N>,
                          rcol_nb(-N), rcol_threads(-N), rcol_smem(-N), nullptr, 0, 0, 0, 0, 0};
    else
        static_assert(N >= 8 && is_pow2(N), "no kernels for this length class");
}

}  // namespace imr
