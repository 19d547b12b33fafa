// Host-side helpers shared by the engine's translation units.
#pragma once
#include <cuda_runtime.h>
#include <vector>
#include "imresh_b200.h"
#include "engine.cuh"
#include "rules.hpp"

namespace imr {

// Launch of a pass; with `dependent` it may start while the pass before it on
// the stream drains (programmatic dependent launch; the kernel calls pdl_wait
// before it touches what earlier passes write).
template <class... P, class... A>
inline cudaError_t launch_pass(bool dependent, void (*kernel)(P...), int grid, int threads, size_t smem, cudaStream_t s,
                               A... args)
{
    if (!dependent) {   // (the plain launch costs less host time in a capture)
        kernel<<<grid, threads, smem, s>>>(static_cast<P>(args)...);
        return cudaGetLastError();
    }
    cudaLaunchConfig_t c{};
    c.gridDim = dim3((unsigned)grid);
    c.blockDim = dim3((unsigned)threads);
    c.dynamicSmemBytes = smem;
    c.stream = s;
    cudaLaunchAttribute a{};
    a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &a;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, kernel, args...);
}

constexpr unsigned kMaxSide = 4096;
constexpr int kMaxRuntimeSide = 2048;

extern thread_local char g_last_error[256];   // imr_last_error() text
void set_error(const char *what, cudaError_t e);
bool factor_len(int n, std::vector<int> &rad);
bool length_supported(int n);
int bluestein_m(int n);
int make_fft_plan(int n, FftPlanDev &p);
int gaussian_weights(double sigma, float *w, int cap);
int ensure_kernel_attributes();
// Scratch of a synchronous call (free with cudaFreeAsync on the same stream).
cudaError_t scratch_alloc(void **p, size_t bytes, cudaStream_t s);
// Give the kept scratch memory of the current device back to the driver.
cudaError_t scratch_release();
// cudaMalloc that gives the kept scratch back and tries again when memory is out.
cudaError_t device_alloc(void **p, size_t bytes);
void resolve_params(const imr_params *in, imr_params &out);
int build_weight_table(const imr_params &p, std::vector<float> &w, std::vector<int> &taps);

// Kernels and launch shape of the row passes for one row length.
struct RowKernels {
    void (*hio_first)(const JobDev *, const WorkList *);
    void (*hio)(const JobDev *, const WorkList *);
    void (*finish)(const JobDev *, const WorkList *, float2 *);
    void (*fft_fwd)(float2 *, FftPlanDev, int, int);
    void (*fft_inv)(float2 *, FftPlanDev, int, int);
    int nb;        // rows per CTA
    int threads;
    int smem;      // dynamic shared memory of the FFT kernels (bytes); 0: nb*N*8
    // pipelined (persistent, TMA) row passes; null when the length has none
    void (*p_hio_first)(const JobDev *, const WorkList *);
    void (*p_hio)(const JobDev *, const WorkList *);
    int p_smem_first, p_smem;
    // fixed-support HIO row passes (libs::hybridInputOutput): per-tile kernel
    // and, where the length has one, the pipelined kernel (shared memory p_smem)
    void (*hio_fix)(const JobDev *, const WorkList *);
    void (*p_hio_fix)(const JobDev *, const WorkList *);
    // pipelined once-per-cycle pass (g', out, error sums, row blur) or null
    void (*p_finish)(const JobDev *, const WorkList *, float2 *);
    int p_smem_fin;
    int mx;        // 1: grouped-pass kernels (kernels_mx.cuh), nb is the most rows of a tile
    // passes of small images (n_nb rows per one-item block), or null
    void (*n_hio_first)(const JobDev *, const WorkList *);
    void (*n_hio)(const JobDev *, const WorkList *);
    void (*n_hio_fix)(const JobDev *, const WorkList *);
    int n_nb, n_threads, n_smem;
};
// Kernels and launch shape of the column passes for one column length.
struct ColKernels {
    void (*col)(const JobDev *, const WorkList *);
    void (*init)(const JobDev *, const WorkList *);
    void (*fft_fwd)(float2 *, FftPlanDev, int, int);
    void (*fft_inv)(float2 *, FftPlanDev, int, int);
    int nb;        // columns per CTA
    int threads;
    int smem;      // dynamic shared memory (bytes); 0: nb*N*8
    void (*p_col)(const JobDev *, const WorkList *);   // pipelined column pass or null
    int p_smem;
    int p_box_rows;  // rows per 2D TMA box
    int p_tma_m;     // 1: the modulus tile also arrives by TMA
    int p_threads;   // threads of the pipelined column pass
    int p_nb;        // columns per tile of the pipelined pass (its TMA box width)
    int p_mt;        // 1: the pipelined pass reads the modulus from JobDev::Mt when set
    // split-precision tensor-core column passes ([0] BF16 hi+lo, [1] FP16 hi+lo;
    // same launch shape as p_col) and their stand-alone forward / inverse
    // column transforms; null where the length has none
    void (*p_col_tc[2])(const JobDev *, const WorkList *);
    void (*fft_tc[2][2])(const JobDev *, const WorkList *);   // [precision][0 forward, 1 inverse]
    int p_smem_tc;   // their dynamic shared memory
    void (*p_col_split)(const JobDev *, const WorkList *);   // p_col running WorkList::n_split
                                                              // tiles as half tiles (JobDev::tmXh), or null
    int checks;      // 1: `col` takes a block more for the deferred error of a fixed-support plan
    void (*f_fwd)(float2 *, FftPlanDev, int, int);   // fft_fwd, fft_inv in narrow tiles, or null
    void (*f_inv)(float2 *, FftPlanDev, int, int);
    int f_nb, f_threads, f_smem;
    void (*n_col)(const JobDev *, const WorkList *);   // pass of small images (n_nb columns per one-item block), or null
    int n_nb, n_threads, n_smem;
};
RowKernels row_kernels(int N);
// Rows per tile of the per-tile row kernels on a W x H image, and the dynamic
// shared memory of such a tile.
int rows_per_tile(const RowKernels &rk, int W, int H);
int row_tile_smem(const RowKernels &rk, int W, int rpc);
// W: columns of the one image of a launch (several images of a launch: many).
constexpr int kManyColumns = 1 << 30;
ColKernels col_kernels(int N, int W = kManyColumns);
// Lengths with kernels specialised at compile time and Bluestein transform
// lengths M (power of two >= 2n - 1 for n <= 2048); any other supported length
// runs the grouped-pass kernels (row_set_mx, col_set_mx).
#define IMR_SIZES(X) X(64) X(128) X(192) X(256) X(384) X(512) X(768) X(1024) X(1536) X(2048) X(3072) X(4096)
#define IMR_BS_SIZES(X) X(-8) X(-16) X(-32) X(-64) X(-128) X(-256) X(-512) X(-1024) X(-2048) X(-4096)
template <int N>
RowKernels row_set();
template <int N>
ColKernels col_set();
RowKernels row_set_mx(int n);
ColKernels col_set_mx(int n, int W);
// Plain 2D transform passes (axes: 1 rows, 2 columns, 3 both).
int fft_passes(float2 *d, int W, int H, int sign, int axes, const FftPlanDev &pr, const FftPlanDev &pc,
               cudaStream_t s);
void narrow_tiles(const RowKernels &rk, const ColKernels &ck, bool p_cols, int W, int H, int *rows, int *cols);
// Persistent grid size for a pipelined kernel (CTAs per SM x SMs, <= items).
int persistent_grid(const void *kernel, int threads, int smem, int items);
// Launch the once-per-cycle row pass over `items` row tiles: the pipelined
// persistent kernel where the row length has one, else one CTA per tile.
// grid_pct: the persistent grid at this percentage of the occupancy limit.
int launch_finish(const RowKernels &rk, int items, size_t smem_fin, cudaStream_t s, const JobDev *dj,
                  const WorkList *L, float2 *dbg, int grid_pct = 100, bool dependent = false);
// Persistent grid scaled to grid_pct % of the occupancy limit (at least 1 CTA, at most `items`).
int scaled_grid(const void *kernel, int threads, int smem, int items, int grid_pct);
// WorkList::n_split of a persistent column launch of n_tiles tiles with at
// most g_max CTAs resident (its grid: min(g_max, n_tiles + n_split)): every
// tile when their halves fit the resident CTAs, else none.
int col_split(int n_tiles, int g_max);
// 2D tensor map over a row-major [H][W] array of `elem`-byte elements with a
// (box_w, box_h) box; returns false when the shape cannot be described.
bool encode_tensor_map(CUtensorMap *map, const void *base, int W, int H, int elem, int box_w, int box_h);

// Host description of one reconstruction's device layout and kernels.
struct JobShape {
    RowKernels rk{};
    ColKernels ck{};
    bool p_rows = false, p_cols = false;
    bool p_half = false;   // JobDev::tmXh encoded: the column pass may run half tiles
    size_t smem_row = 0, smem_fin = 0, smem_col = 0;
    size_t bytes = 0;   // arena bytes (JobState not included)
    size_t oX = 0, oG = 0, oM = 0, oMt = 0, oHB = 0, oVB = 0, oOut = 0, oMask = 0, oW = 0, oT = 0, oEP = 0, oErr = 0;
    std::vector<float> wt;
    std::vector<int> taps;
};
bool passes_dependent(const JobDev &J, const JobShape &S, const RowKernels &rk, const ColKernels &ck, bool fix, int n_split,
                      bool row_narrow, bool col_narrow);
// alone: no launch holds passes of other jobs.
int job_prepare(unsigned W, unsigned H, const imr_params &p, JobDev &J, JobShape &S, bool alone = true);
void job_bind(JobDev &J, JobShape &S, char *arena, JobState *st);
int job_upload(const JobDev &J, const JobShape &S, char *arena, JobDev *dj, cudaStream_t s);
// Fill JobDev::Mt from the modulus (stream-ordered; nothing to do when Mt is
// null).  Called whenever the modulus has been (re)written.
int job_modulus_tiles(const JobDev &J, cudaStream_t s);
int plan_cache_acquire(unsigned W, unsigned H, const imr_params *params, imr_plan **out);
void plan_cache_release(imr_plan *P);

}  // namespace imr
