// Host side of the engine: FFT plans, reconstruction plans (device buffers +
// captured CUDA graph of one shrink-wrap cycle) and the C ABI declared in
// include/imresh_b200.h.
#include <cuda_runtime.h>
#include <float.h>
#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

#include "imresh_b200.h"
#include "kernels.cuh"
#include "engine_host.hpp"
#include <cudaTypedefs.h>

namespace imr {

thread_local char g_last_error[256] = "";

void set_error(const char *what, cudaError_t e)
{
    snprintf(g_last_error, sizeof(g_last_error), "%s: %s", what, cudaGetErrorString(e));
}

// ---------------------------------------------------------------- lengths
// Radix schedule: 8s first (4,4 or 4 or 2 for the remaining power of two),
// then 3s, 5s and 7s.  Supported lengths: every 2^a 3^b 5^c 7^d up to
// kMaxRuntimeSide (runtime-length kernels hold 8 values x 256 threads), and
// the compile-time lengths 3072 and 4096 above it.
bool factor_len(int n, std::vector<int> &rad)
{
    rad.clear();
    if (n < 1 || n > (int)kMaxSide) return false;
    if (n > kMaxRuntimeSide && n != 3072 && n != 4096) return false;
    int m = n, k = 0;
    while (m % 2 == 0) { m /= 2; ++k; }
    while (k >= 3 && !(k == 4)) { rad.push_back(8); k -= 3; }
    if (k == 4) { rad.push_back(4); rad.push_back(4); }
    else if (k == 2) rad.push_back(4);
    else if (k == 1) rad.push_back(2);
    for (int p : {3, 5, 7})
        while (m % p == 0) { rad.push_back(p); m /= p; }
    return m == 1 && (int)rad.size() <= 14;
}

// Supported image sides: every length 1..kMaxRuntimeSide (direct mixed-radix
// transforms when the length factors into 2, 3, 5, 7; Bluestein otherwise),
// plus the compile-time lengths 3072 and 4096.
int bluestein_m(int n)
{
    int m = 1;
    while (m < 2 * n - 1) m <<= 1;
    return m;
}

bool length_supported(int n)
{
    std::vector<int> rad;
    if (factor_len(n, rad)) return true;
    return n >= 1 && n <= kMaxRuntimeSide;
}

// in-place radix-2 FFT in double (host; Bluestein kernel spectra)
static void host_fft_pow2(std::vector<double> &re, std::vector<double> &im, int sign)
{
    const int n = (int)re.size();
    for (int i = 1, j = 0; i < n; ++i) {
        int bit = n >> 1;
        for (; j & bit; bit >>= 1) j ^= bit;
        j ^= bit;
        if (i < j) {
            std::swap(re[i], re[j]);
            std::swap(im[i], im[j]);
        }
    }
    for (int len = 2; len <= n; len <<= 1) {
        for (int i = 0; i < n; i += len)
            for (int k = 0; k < len / 2; ++k) {
                const double a = sign * 2.0 * M_PI * (double)k / (double)len;
                const double wr = cos(a), wi = sin(a);
                const double ur = re[i + k], ui = im[i + k];
                const double xr = re[i + k + len / 2], xi = im[i + k + len / 2];
                const double vr = xr * wr - xi * wi, vi = xr * wi + xi * wr;
                re[i + k] = ur + vr;
                im[i + k] = ui + vi;
                re[i + k + len / 2] = ur - vr;
                im[i + k + len / 2] = ui - vi;
            }
    }
}

// Twiddle tables exp(-2 pi i t/L), t < L, computed in double; one per
// (device, n), kept for the life of the process.  Bluestein lengths also
// keep their chirp and kernel spectra in the same allocation.
static std::mutex g_tw_mu;
static std::map<std::pair<int, int>, float2 *> g_tw;

static int make_bluestein_plan(int n, FftPlanDev &p)
{
    const int M = bluestein_m(n);
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(g_tw_mu);
    auto key = std::make_pair(dev, -n);
    float2 *d = nullptr;
    auto it = g_tw.find(key);
    if (it == g_tw.end()) {
        std::vector<float2> h((size_t)M + n + 2 * (size_t)M);
        for (int t = 0; t < M; ++t) {
            const double a = -2.0 * M_PI * (double)t / (double)M;
            h[t] = make_float2((float)cos(a), (float)sin(a));
        }
        std::vector<double> cre(n), cim(n);
        for (int j = 0; j < n; ++j) {
            const long long q = ((long long)j * j) % (2LL * n);   // j^2 mod 2n: exact angle
            const double a = -M_PI * (double)q / (double)n;
            cre[j] = cos(a);
            cim[j] = sin(a);
            h[M + j] = make_float2((float)cre[j], (float)cim[j]);
        }
        for (int dir = 0; dir < 2; ++dir) {   // 0: forward (S = -1), 1: inverse (S = +1)
            std::vector<double> kr(M, 0.0), ki(M, 0.0);
            for (int j = 0; j < n; ++j) {
                // kernel conj(c_j) with c_j = exp(S i pi j^2/n), wrapped for negative j
                const double br = cre[j], bi = dir == 0 ? -cim[j] : cim[j];
                kr[j] = br;
                ki[j] = bi;
                if (j) {
                    kr[M - j] = br;
                    ki[M - j] = bi;
                }
            }
            host_fft_pow2(kr, ki, -1);
            for (int t = 0; t < M; ++t)
                h[(size_t)M + n + (size_t)dir * M + t] = make_float2((float)(kr[t] / M), (float)(ki[t] / M));
        }
        cudaError_t e = cudaMalloc(&d, sizeof(float2) * h.size());
        if (e != cudaSuccess) { set_error("cudaMalloc Bluestein tables", e); return IMR_ERR_OUT_OF_MEMORY; }
        e = cudaMemcpy(d, h.data(), sizeof(float2) * h.size(), cudaMemcpyHostToDevice);
        if (e != cudaSuccess) { set_error("cudaMemcpy Bluestein tables", e); return IMR_ERR_CUDA; }
        g_tw[key] = d;
    } else {
        d = it->second;
    }
    memset(&p, 0, sizeof(p));
    p.n = n;
    p.bs_m = M;
    p.tw = d;
    p.chirp = d + M;
    p.bspec_f = d + M + n;
    p.bspec_b = d + M + n + M;
    return IMR_SUCCESS;
}

int make_fft_plan(int n, FftPlanDev &p)
{
    std::vector<int> rad;
    if (!factor_len(n, rad)) return length_supported(n) ? make_bluestein_plan(n, p) : IMR_ERR_UNSUPPORTED_SIZE;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(g_tw_mu);
    auto key = std::make_pair(dev, n);
    auto it = g_tw.find(key);
    float2 *d = nullptr;
    if (it == g_tw.end()) {
        std::vector<float2> h(n);
        for (int t = 0; t < n; ++t) {
            double a = -2.0 * M_PI * (double)t / (double)n;
            h[t] = make_float2((float)cos(a), (float)sin(a));
        }
        cudaError_t e = cudaMalloc(&d, sizeof(float2) * n);
        if (e != cudaSuccess) { set_error("cudaMalloc twiddles", e); return IMR_ERR_OUT_OF_MEMORY; }
        e = cudaMemcpy(d, h.data(), sizeof(float2) * n, cudaMemcpyHostToDevice);
        if (e != cudaSuccess) { set_error("cudaMemcpy twiddles", e); return IMR_ERR_CUDA; }
        g_tw[key] = d;
    } else {
        d = it->second;
    }
    memset(&p, 0, sizeof(p));
    p.n = n;
    p.nrad = (int)rad.size();
    for (size_t i = 0; i < rad.size(); ++i) p.rad[i] = rad[i];
    fft_group_passes(p);
    p.tw = d;
    return IMR_SUCCESS;
}

// calcGaussianKernel<float> (src/imresh/libs/calcGaussianKernel.cpp:42-91):
// half width ceil(2.884402748387961466*sigma - 0.5); weights a*exp(i*i*b)
// rounded to float, normalised by their double sum.
int gaussian_weights(double sigma, float *w, int cap)
{
    const int half = (int)ceil(2.884402748387961466 * sigma - 0.5);
    const int K = 2 * half + 1;
    if (w == nullptr || K > cap) return K;
    const double a = 1.0 / (sqrt(2.0 * M_PI) * sigma);
    const double b = -1.0 / (2.0 * sigma * sigma);
    double sum = 0;
    for (int i = -half; i <= half; ++i) {
        float v = (float)(a * exp(i * i * b));
        w[half + i] = v;
        sum += v;
    }
    for (int i = 0; i < K; ++i) w[i] = (float)((double)w[i] / sum);
    return K;
}

// ---------------------------------------------------------------- scratch memory
// Device memory of the synchronous host-buffer calls (forward model, maximum,
// error): from one pool per device that keeps up to kScratchKeep bytes between
// calls and gives the rest back.  The default pool gives everything back at each
// synchronisation, and mapping it again took half of a 1000 x 800 forward model
// (0.5 of 1.0 ms).  Stream-ordered, so calls on several streams and threads may
// overlap.  What it keeps is given back before an engine counts the free memory,
// when an allocation of a plan or a request fails, and by imr_release_scratch.
constexpr uint64_t kScratchKeep = 256ull << 20;
static std::mutex g_pool_mu;
static std::map<int, cudaMemPool_t> g_pool;

cudaError_t scratch_alloc(void **p, size_t bytes, cudaStream_t s)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    cudaMemPool_t pool = nullptr;
    {
        std::lock_guard<std::mutex> lk(g_pool_mu);
        auto it = g_pool.find(dev);
        if (it == g_pool.end()) {
            cudaMemPoolProps pp;
            memset(&pp, 0, sizeof(pp));
            pp.allocType = cudaMemAllocationTypePinned;
            pp.handleTypes = cudaMemHandleTypeNone;
            pp.location.type = cudaMemLocationTypeDevice;
            pp.location.id = dev;
            uint64_t keep = kScratchKeep;
            e = cudaMemPoolCreate(&pool, &pp);
            if (e == cudaSuccess) e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
            if (e != cudaSuccess) {
                if (pool) cudaMemPoolDestroy(pool);
                return e;
            }
            g_pool[dev] = pool;
        } else {
            pool = it->second;
        }
    }
    return cudaMallocFromPoolAsync(p, bytes, pool, s);
}

cudaError_t scratch_release()
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lk(g_pool_mu);
    auto it = g_pool.find(dev);
    return it == g_pool.end() ? cudaSuccess : cudaMemPoolTrimTo(it->second, 0);
}

cudaError_t device_alloc(void **p, size_t bytes)
{
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaErrorMemoryAllocation) return e;
    cudaGetLastError();
    e = scratch_release();
    return e == cudaSuccess ? cudaMalloc(p, bytes) : e;
}

// ---------------------------------------------------------------- dispatch
// Resident CTAs per SM of a kernel at a launch shape, asked of the occupancy
// calculator once per (device, kernel, shape): the engine launches hundreds
// of persistent passes per step.
struct OccKey {
    int dev;
    const void *k;
    int threads, smem;
    bool operator<(const OccKey &o) const
    {
        return std::tie(dev, k, threads, smem) < std::tie(o.dev, o.k, o.threads, o.smem);
    }
};
static std::mutex g_occ_mu;
static std::map<OccKey, std::pair<int, int>> g_occ;   // -> (CTAs per SM, SMs)

int persistent_grid(const void *kernel, int threads, int smem, int items)
{
    int dev = 0;
    cudaGetDevice(&dev);
    const OccKey key{dev, kernel, threads, smem};
    std::pair<int, int> occ;
    {
        std::lock_guard<std::mutex> lk(g_occ_mu);
        auto it = g_occ.find(key);
        if (it != g_occ.end()) {
            occ = it->second;
        } else {
            int sms = 148, per_sm = 1;
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess ||
                per_sm < 1)
                per_sm = 1;
            occ = {per_sm, sms};
            g_occ[key] = occ;
        }
    }
    const long g = (long)occ.first * occ.second;
    return (int)(g < items ? g : items);
}

// Tiles of the small-image passes for a W x H plan, 0 where they are not used:
// up to 1024 sequences of up to 1024 values (HIO iteration, pipelined passes ->
// these, both launched dependently: 64^2 6.5 -> 4.7 us, 256^2 8.1 -> 6.1, 384^2 14.4 ->
// 8.3, 512^2 11.6 -> 8.4, 1024^2 20.1 -> 16.7).  Beyond that their tiles are many
// and the pipelined passes' copies ahead pay again (2048 columns of 512: 10.1 us
// against 11.3; 2048 rows of 512: 8.9 against 11.0).  They replace pipelined
// passes only: the per-tile passes of other shapes (widths that no tensor map
// describes) order their transforms differently.
void narrow_tiles(const RowKernels &rk, const ColKernels &ck, bool p_cols, int W, int H, int *rows, int *cols)
{
    *rows = rk.n_hio && H <= 1024 ? (H + rk.n_nb - 1) / rk.n_nb : 0;
    *cols = ck.n_col && p_cols && W <= 1024 ? (W + ck.n_nb - 1) / ck.n_nb : 0;
}

// Whether the two passes of an iteration on a W x H job are launched dependently
// (see dependent_pass; the small-image passes always may be: one short item per
// block, placed as SMs become free).
bool passes_dependent(const JobDev &J, const JobShape &S, const RowKernels &rk, const ColKernels &ck, bool fix, int n_split,
                      bool row_narrow, bool col_narrow)
{
    const int every = 1 << 30;
    auto row_ok = [&] {
        const auto pk = fix ? rk.p_hio_fix : rk.p_hio;
        const auto k = fix ? rk.hio_fix : rk.hio;
        return dependent_pass(J.n_row_tiles, pk ? persistent_grid((const void *)pk, rk.threads, rk.p_smem, every)
                                                : persistent_grid((const void *)k, rk.threads, (int)S.smem_row, every));
    };
    auto col_ok = [&] {
        return S.p_cols ? dependent_pass(J.n_col_tiles + n_split,
                                         persistent_grid((const void *)ck.p_col, ck.p_threads, ck.p_smem, every))
                        : dependent_pass(J.n_col_tiles,
                                         persistent_grid((const void *)ck.col, ck.threads, (int)S.smem_col, every));
    };
    if (!row_narrow && rk.p_hio && !pipelined_rows_dependent(J.W)) return false;
    return (row_narrow || row_ok()) && (col_narrow || col_ok());
}

// A persistent column pass runs one tile per CTA at a time.  When the tiles
// fill at most half of the resident CTAs (256^2: 16 tiles, 512^2: 32, on 148
// SMs) every tile runs as two half tiles on two CTAs (bit-identical results):
// measured 5.6 -> 5.1 us at 256^2 and 8.8 -> 6.9 us at 512^2.  Beyond that a
// half tile, at ~79 % of a whole tile's time, loses: splitting each CTA's first
// and last tile at 2048^2 took the pass from 33.3 to 37.6 us, and all tiles at
// 1024^2 (two rounds of halves) from 9.8 to 12.7 us.
int col_split(int n_tiles, int g_max)
{
    return (n_tiles > 0 && 2 * n_tiles <= g_max) ? n_tiles : 0;
}

int scaled_grid(const void *kernel, int threads, int smem, int items, int grid_pct)
{
    const int g = persistent_grid(kernel, threads, smem, 1 << 30);   // the occupancy limit
    const long want = std::max(1L, (long)g * grid_pct / 100);
    return (int)std::min<long>(want, std::max(items, 1));
}

int launch_finish(const RowKernels &rk, int items, size_t smem_fin, cudaStream_t s, const JobDev *dj,
                  const WorkList *L, float2 *dbg, int grid_pct, bool dependent)
{
    const cudaError_t e =
        rk.p_finish ? launch_pass(dependent, rk.p_finish,
                                  scaled_grid((const void *)rk.p_finish, rk.threads, rk.p_smem_fin, items, grid_pct),
                                  rk.threads, rk.p_smem_fin, s, dj, L, dbg)
                    : launch_pass(dependent, rk.finish, items, rk.threads, smem_fin, s, dj, L, dbg);
    if (e != cudaSuccess) {
        set_error("finish launch", e);
        return IMR_ERR_CUDA;
    }
    return IMR_SUCCESS;
}

static PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;

bool encode_tensor_map(CUtensorMap *map, const void *base, int W, int H, int elem, int box_w, int box_h)
{
    if (!g_encode) {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess || !fn)
            return false;
        g_encode = (PFN_cuTensorMapEncodeTiled_v12000)fn;
    }
    if (((size_t)W * elem) % 16 != 0 || ((uintptr_t)base & 15) != 0 || (box_w * elem) % 16 != 0) return false;
    if (box_w > 256 || box_h > 256 || box_w > W || box_h > H) return false;
    cuuint64_t dims[2] = {(cuuint64_t)W, (cuuint64_t)H};
    cuuint64_t strides[1] = {(cuuint64_t)W * elem};
    cuuint32_t box[2] = {(cuuint32_t)box_w, (cuuint32_t)box_h};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = g_encode(map, elem == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2,
                          const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

RowKernels row_kernels(int N)
{
    std::vector<int> rad;
    if (!factor_len(N, rad) && length_supported(N)) N = -bluestein_m(N);
    switch (N) {
#define ROWCASE(n) case n: return row_set<n>();
        IMR_SIZES(ROWCASE)
        IMR_BS_SIZES(ROWCASE)
#undef ROWCASE
    default: return row_set_mx(N);
    }
}

// The grouped-pass kernels take as few rows per tile as give every SM three
// tiles (148 x 3), but at least 512 values (two per thread); the others a fixed
// number.
int rows_per_tile(const RowKernels &rk, int W, int H)
{
    const int most = std::min(rk.nb, H);
    return rk.mx ? std::min(most, std::max((H + 443) / 444, (511 + W) / W)) : most;
}
int row_tile_smem(const RowKernels &rk, int W, int rpc) { return rk.mx ? mx_row_smem(W, rpc) : rk.smem; }

ColKernels col_kernels(int N, int W)
{
    std::vector<int> rad;
    if (!factor_len(N, rad) && length_supported(N)) N = -bluestein_m(N);
    switch (N) {
#define COLCASE(n) case n: return col_set<n>();
        IMR_SIZES(COLCASE)
        IMR_BS_SIZES(COLCASE)
#undef COLCASE
    default: return col_set_mx(N, W);
    }
}

static std::mutex g_attr_mu;
static std::vector<int> g_attr_done;

// Opt every kernel into the device's largest dynamic shared-memory size
// (opt-in limit minus the kernel's static shared memory).
static int g_optin_smem = 0;

template <class F>
static cudaError_t allow_smem(F f)
{
    cudaFuncAttributes fa;
    cudaError_t e = cudaFuncGetAttributes(&fa, (const void *)f);
    if (e != cudaSuccess) return e;
    const int dyn = g_optin_smem - (int)fa.sharedSizeBytes;
    return cudaFuncSetAttribute((const void *)f, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn);
}

int ensure_kernel_attributes()
{
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(g_attr_mu);
    for (int d : g_attr_done)
        if (d == dev) return IMR_SUCCESS;
    cudaError_t e = cudaDeviceGetAttribute(&g_optin_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    std::vector<int> sizes = {5, 2000};   // lengths of the grouped-pass kernels of either column width
#define PUSH(n) sizes.push_back(n);
    IMR_SIZES(PUSH)
#undef PUSH
    std::vector<RowKernels> rks;
    std::vector<ColKernels> cks;
    for (int n : sizes) {
        rks.push_back(row_kernels(n));
        cks.push_back(col_kernels(n));
    }
    rks.push_back(rks.front());   // (a pair for the few-column kernels)
    cks.push_back(col_kernels(2000, 1));
#define PUSHBS(n) rks.push_back(row_set<n>()); cks.push_back(col_set<n>());
    IMR_BS_SIZES(PUSHBS)
#undef PUSHBS
    for (size_t q = 0; q < rks.size(); ++q) {
        RowKernels r = rks[q];
        ColKernels c = cks[q];
        if (e == cudaSuccess) e = allow_smem(r.hio_first);
        if (e == cudaSuccess) e = allow_smem(r.hio);
        if (e == cudaSuccess) e = allow_smem(r.finish);
        if (e == cudaSuccess) e = allow_smem(r.fft_fwd);
        if (e == cudaSuccess) e = allow_smem(r.fft_inv);
        if (e == cudaSuccess) e = allow_smem(c.col);
        if (e == cudaSuccess) e = allow_smem(c.init);
        if (e == cudaSuccess) e = allow_smem(c.fft_fwd);
        if (e == cudaSuccess) e = allow_smem(c.fft_inv);
        if (e == cudaSuccess && c.f_fwd) e = allow_smem(c.f_fwd);
        if (e == cudaSuccess && c.f_inv) e = allow_smem(c.f_inv);
        if (e == cudaSuccess && r.p_hio) e = allow_smem(r.p_hio);
        if (e == cudaSuccess && r.p_hio_first) e = allow_smem(r.p_hio_first);
        if (e == cudaSuccess) e = allow_smem(r.hio_fix);
        if (e == cudaSuccess && r.n_hio) e = allow_smem(r.n_hio);
        if (e == cudaSuccess && r.n_hio) e = allow_smem(r.n_hio_first);
        if (e == cudaSuccess && r.n_hio) e = allow_smem(r.n_hio_fix);
        if (e == cudaSuccess && c.n_col) e = allow_smem(c.n_col);
        if (e == cudaSuccess && r.p_hio_fix) e = allow_smem(r.p_hio_fix);
        if (e == cudaSuccess && r.p_finish) e = allow_smem(r.p_finish);
        if (e == cudaSuccess && c.p_col) e = allow_smem(c.p_col);
        if (e == cudaSuccess && c.p_col_split) e = allow_smem(c.p_col_split);
        for (int pr = 0; pr < 2; ++pr) {
            if (e == cudaSuccess && c.p_col_tc[pr]) e = allow_smem(c.p_col_tc[pr]);
            for (int d = 0; d < 2; ++d)
                if (e == cudaSuccess && c.fft_tc[pr][d]) e = allow_smem(c.fft_tc[pr][d]);
        }
    }
    if (e == cudaSuccess) e = allow_smem(k_hblur<true>);
    if (e == cudaSuccess) e = allow_smem(k_hblur<false>);
    if (e == cudaSuccess) e = allow_smem(k_hblur_px);
    if (e != cudaSuccess) {
        set_error("cudaFuncSetAttribute", e);
        return IMR_ERR_CUDA;
    }
    g_attr_done.push_back(dev);
    return IMR_SUCCESS;
}

void resolve_params(const imr_params *in, imr_params &p)
{
    // Defaults of the reference's CUDA driver (cudaShrinkWrap.cu:193-200).
    if (in) p = *in;
    else memset(&p, 0, sizeof(p));
    if (p.nCycles == 0) p.nCycles = 20;
    if (!(p.targetError > 0)) p.targetError = 1e-5f;
    if (!(p.hioBeta > 0)) p.hioBeta = 0.9f;
    if (!(p.intensityCutOffAutoCorel > 0)) p.intensityCutOffAutoCorel = 0.02f;
    if (!(p.intensityCutOff > 0)) p.intensityCutOff = 0.2f;
    if (!(p.sigma0 > 0)) p.sigma0 = 3.0f;
    if (!(p.sigmaChange > 0)) p.sigmaChange = 0.01f;
    if (p.nHioCycles == 0) p.nHioCycles = 20;
}

// Sigma of every cycle (sigma <- max(1.5, (1 - change)*sigma) after each
// mask, in float: cudaShrinkWrap.cu:294) and its Gaussian weights.  Entry
// n_cycles serves the final error-only pass.
int build_weight_table(const imr_params &p, std::vector<float> &w, std::vector<int> &taps)
{
    w.assign((size_t)(p.nCycles + 1) * kTapStride, 0.f);
    taps.assign(p.nCycles + 1, 1);
    float sigma = p.sigma0;
    for (unsigned c = 0; c <= p.nCycles; ++c) {
        int K = gaussian_weights((double)sigma, &w[(size_t)c * kTapStride], kMaxTaps);
        if (K > kMaxTaps) return IMR_ERR_INVALID_VALUE;
        taps[c] = K;
        sigma = fmaxf(1.5f, (1.0f - p.sigmaChange) * sigma);
    }
    return IMR_SUCCESS;
}

// Unnormalised 2D transform passes over a [H][W] complex array with the
// plain FFT kernels: axes bit 1 = rows, bit 2 = columns; sign -1 runs rows
// then columns, +1 columns then rows.
static int fft_launch(float2 *d, int W, int H, int sign, int axes, const FftPlanDev &pr, const FftPlanDev &pc,
                      const RowKernels &rk, const ColKernels &ck, cudaStream_t s)
{
    const int every = 1 << 30, wide = (W + ck.nb - 1) / ck.nb;
    const bool narrow = ck.f_fwd && (fft_narrow_columns(wide) ||   // (asks only where the count does not decide)
                                     fft_narrow_columns(wide, persistent_grid((const void *)ck.fft_fwd, ck.threads, ck.smem, every)));
    const int rpc = rk.mx ? rows_per_tile(rk, W, H) : rk.nb, cpc = narrow ? ck.f_nb : ck.nb;
    const int nrt = (H + rpc - 1) / rpc, nct = (W + cpc - 1) / cpc, ct = narrow ? ck.f_threads : ck.threads;
    const size_t sr = rk.smem ? (size_t)row_tile_smem(rk, W, rpc) : (size_t)rpc * W * 8;
    const size_t sc = narrow ? (size_t)ck.f_smem : ck.smem ? (size_t)ck.smem : (size_t)H * cpc * 8;
    const auto rows = sign < 0 ? rk.fft_fwd : rk.fft_inv;
    const auto cols = sign < 0 ? (narrow ? ck.f_fwd : ck.fft_fwd) : (narrow ? ck.f_inv : ck.fft_inv);
    // the second transform may start while the first one drains (fft_rows_start_early)
    auto rows_early = [&] {
        if (nrt <= 111 || !rk.p_hio) return true;   // (few, or grouped or chirp-z rows: nothing to ask)
        const int cols_resident = persistent_grid((const void *)cols, ct, (int)sc, every);
        return fft_rows_start_early(nct, cols_resident, nrt, persistent_grid((const void *)rows, rk.threads, (int)sr, every),
                                    is_pow2(W) && is_pow2(H) && cols_resident > kSms);
    };
    const bool dep = axes == 3 && (sign < 0 || rows_early());
    cudaError_t e = cudaSuccess;
    if (sign < 0) {
        if (axes & 1) e = launch_pass(false, rows, nrt, rk.threads, sr, s, d, pr, H, rpc);
        if ((axes & 2) && e == cudaSuccess) e = launch_pass(dep, cols, nct, ct, sc, s, d, pc, W, cpc);
    } else {
        if (axes & 2) e = launch_pass(false, cols, nct, ct, sc, s, d, pc, W, cpc);
        if ((axes & 1) && e == cudaSuccess) e = launch_pass(dep, rows, nrt, rk.threads, sr, s, d, pr, H, rpc);
    }
    if (e != cudaSuccess) {
        set_error("fft launch", e);
        return IMR_ERR_CUDA;
    }
    return IMR_SUCCESS;
}
int fft_passes(float2 *d, int W, int H, int sign, int axes, const FftPlanDev &pr, const FftPlanDev &pc,
               cudaStream_t s)
{
    return fft_launch(d, W, H, sign, axes, pr, pc, row_kernels(W), col_kernels(H, W), s);
}

}  // namespace imr

using namespace imr;

// ==================================================================== plans
constexpr int kPlanGraphCycles = 64;   // shrink-wrap cycles per captured graph

struct imr_plan {
    int dev = 0;
    int W = 0, H = 0;
    imr_params p{};
    JobDev hj{};
    JobDev *dj = nullptr;
    JobState *st = nullptr;
    void *arena = nullptr;
    size_t smem_row = 0, smem_fin = 0, smem_col = 0;
    // the cycles of one execution as at most two captured graphs: `chunk`
    // cycles replayed n_chunks times, then the remaining cycles
    cudaGraphExec_t gexec = nullptr, gexec_rem = nullptr;
    cudaGraph_t graph = nullptr, graph_rem = nullptr;
    int chunk = 0, n_chunks = 0;
    float2 *dbg_gprime = nullptr;
    RowKernels rk{};
    ColKernels ck{};
    bool p_rows = false, p_cols = false;   // pipelined passes in use
    int g_row_first = 0, g_row = 0, g_col = 0;
    WorkList *Lrow = nullptr, *Lcol = nullptr, *Lvb = nullptr;   // device
    int n_row_narrow = 0, n_col_narrow = 0;       // tiles of the small-image passes (0: not used)
    WorkList *Lrow_n = nullptr, *Lcol_n = nullptr;
    int prec = 0;   // column pass: 0 FP32, 1 BF16 hi+lo tensor cores, 2 FP16 hi+lo tensor cores
    int g_col_tc = 0;
    void (*vblur)(const JobDev *, const WorkList *) = k_vblur<kVbTileY>;
    bool dependent = false;   // passes launched to start while the pass before drains
    bool cols_dependent = false;   // the column passes too
};

// The pipelined column pass of the plan's precision.
static void (*plan_col_kernel(const imr_plan *P))(const JobDev *, const WorkList *)
{
    return P->prec ? P->ck.p_col_tc[P->prec - 1] : P->ck.p_col;
}

// The plan's row and column pass of one HIO iteration.
static cudaError_t plan_launch_row(imr_plan *P, bool first, cudaStream_t s)
{
    const RowKernels &rk = P->rk;
    const JobDev *dj = P->dj;
    const WorkList *L = P->Lrow;
    if (P->n_row_narrow)
        return launch_pass(P->dependent, first ? rk.n_hio_first : rk.n_hio, P->n_row_narrow, rk.n_threads, rk.n_smem, s,
                           dj, (const WorkList *)P->Lrow_n);
    if (!P->p_rows)
        return launch_pass(P->dependent, first ? rk.hio_first : rk.hio, P->hj.n_row_tiles, rk.threads, P->smem_row, s, dj,
                           L);
    return first ? launch_pass(P->dependent, rk.p_hio_first, P->g_row_first, rk.threads, rk.p_smem_first, s, dj, L)
                 : launch_pass(P->dependent, rk.p_hio, P->g_row, rk.threads, rk.p_smem, s, dj, L);
}
static cudaError_t plan_launch_col(imr_plan *P, cudaStream_t s)
{
    const ColKernels &ck = P->ck;
    const JobDev *dj = P->dj;
    const WorkList *L = P->Lcol;
    if (P->prec) return launch_pass(false, plan_col_kernel(P), P->g_col_tc, ck.p_threads, ck.p_smem_tc, s, dj, L);
    if (P->n_col_narrow)
        return launch_pass(P->cols_dependent, ck.n_col, P->n_col_narrow, ck.n_threads, ck.n_smem, s, dj,
                           (const WorkList *)P->Lcol_n);
    if (!P->p_cols) return launch_pass(P->cols_dependent, ck.col, P->hj.n_col_tiles, ck.threads, P->smem_col, s, dj, L);
    return launch_pass(P->cols_dependent, plan_col_kernel(P), P->g_col, ck.p_threads, ck.p_smem, s, dj, L);
}

static int plan_launch_cycle(imr_plan *P, cudaStream_t s)
{
    const JobDev &J = P->hj;
    const RowKernels &rk = P->rk;
    const JobDev *dj = P->dj;
    const WorkList *Lrow = P->Lrow, *Lvb = P->Lvb;
    const bool dep = P->dependent;
    int rc = launch_finish(rk, J.n_row_tiles, P->smem_fin, s, dj, Lrow, P->dbg_gprime, 100, dep);
    if (rc) return rc;
    cudaError_t e = launch_pass(dep, P->vblur, J.n_vb_tiles, kVbThreads, 0, s, dj, Lvb);
    for (int i = 0; i < J.n_hio && e == cudaSuccess; ++i) {
        e = plan_launch_row(P, i == 0, s);
        if (e == cudaSuccess) e = plan_launch_col(P, s);
    }
    if (e != cudaSuccess) {
        set_error("kernel launch", e);
        return IMR_ERR_CUDA;
    }
    return IMR_SUCCESS;
}

#define CK(call)                                  \
    do {                                          \
        cudaError_t e_ = (call);                  \
        if (e_ != cudaSuccess) {                  \
            set_error(#call, e_);                 \
            return IMR_ERR_CUDA;                  \
        }                                         \
    } while (0)

namespace imr {

// ---------------------------------------------------------------- one job
// Host description of one reconstruction's device layout (shared by plans
// and the batched engine).  Arena layout, 256-byte aligned pieces:
// X, G (c64) | M, hb, vb, out (f32) | mask (u8) | weights | taps | error
// partials | per-cycle errors.  The JobState lives wherever the caller puts
// it (plans: after the arena; the engine: in one array for all jobs).
int job_prepare(unsigned W, unsigned H, const imr_params &p, JobDev &J, JobShape &S, bool alone)
{
    int rc;
    memset(&J, 0, sizeof(J));
    J.W = (int)W;
    J.H = (int)H;
    if ((rc = make_fft_plan((int)W, J.prow)) || (rc = make_fft_plan((int)H, J.pcol))) return rc;
    if ((rc = build_weight_table(p, S.wt, S.taps))) return rc;
    S.rk = row_kernels(J.W);
    S.ck = col_kernels(J.H, alone ? J.W : kManyColumns);
    J.rpc = rows_per_tile(S.rk, J.W, J.H);
    J.cpc = S.ck.nb < J.W ? S.ck.nb : J.W;
    S.p_rows = S.rk.p_hio != nullptr;
    S.p_cols = S.ck.p_col != nullptr && J.W % 4 == 0 && J.W >= S.ck.p_nb;
    if (S.p_cols) J.cpc = S.ck.p_nb;
    J.n_row_tiles = (J.H + J.rpc - 1) / J.rpc;
    J.n_col_tiles = (J.W + J.cpc - 1) / J.cpc;
    J.vb_tiles_x = (J.W + kVbTileX - 1) / kVbTileX;
    J.n_vb_tiles = J.vb_tiles_x * ((J.H + kVbTileY - 1) / kVbTileY);
    J.beta = p.hioBeta;
    J.cut_auto = p.intensityCutOffAutoCorel;
    J.cut = p.intensityCutOff;
    J.target = p.targetError;
    J.n_cycles = (int)p.nCycles;
    J.n_hio = (int)p.nHioCycles;
    // shared memory sized for the compile-time tile (NB sequences), even when
    // the image has fewer rows / columns than NB
    if (S.rk.smem) {
        S.smem_row = S.smem_fin = (size_t)row_tile_smem(S.rk, J.W, J.rpc);   // norms reuse the FFT buffers
    } else {
        S.smem_row = (size_t)S.rk.nb * J.W * sizeof(float2);
        S.smem_fin = S.smem_row + (size_t)S.rk.nb * J.W * sizeof(float);
    }
    S.smem_col = S.ck.smem ? (size_t)S.ck.smem
                           : (size_t)S.ck.nb * J.H * sizeof(float2);
    const size_t N = (size_t)W * H;
    auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
    size_t off = 0;
    S.oX = off; off += al(N * 8);
    S.oG = off; off += al(N * 8);
    S.oM = off; off += al(N * 4);
    if (S.p_cols && S.ck.p_mt) {
        S.oMt = off;
        off += al((size_t)((W + S.ck.p_nb - 1) / S.ck.p_nb) * S.ck.p_nb * H * 4);
    }
    S.oHB = off; off += al(N * 4);
    S.oVB = off; off += al(N * 4);
    S.oOut = off; off += al(N * 4);
    S.oMask = off; off += al(N);
    S.oW = off; off += al(S.wt.size() * 4);
    S.oT = off; off += al(S.taps.size() * 4);
    const int n_ep = std::max(J.n_row_tiles, S.rk.n_nb ? (J.H + S.rk.n_nb - 1) / S.rk.n_nb : 0);
    S.oEP = off; off += al((size_t)2 * n_ep * 8);
    S.oErr = off; off += al((size_t)(J.n_cycles + 1) * 4);
    S.bytes = off;
    return IMR_SUCCESS;
}

void job_bind(JobDev &J, JobShape &S, char *a, JobState *st)
{
    J.X = (float2 *)(a + S.oX);
    J.G = (float2 *)(a + S.oG);
    J.M = (const float *)(a + S.oM);
    J.Mt = nullptr;
    J.hb = (float *)(a + S.oHB);
    J.vb = (float *)(a + S.oVB);
    J.out = (float *)(a + S.oOut);
    J.mask = (uint8_t *)(a + S.oMask);
    J.weights = (const float *)(a + S.oW);
    J.ntaps = (const int *)(a + S.oT);
    J.err_part = (double *)(a + S.oEP);
    J.errors = (float *)(a + S.oErr);
    J.st = st;
    J.use_tma_cols = 0;
    if (S.p_cols) {
        const int br = S.ck.p_box_rows;
        bool okm = encode_tensor_map(&J.tmX, J.X, J.W, J.H, 8, S.ck.p_nb, br);
        if (okm && S.ck.p_tma_m) okm = encode_tensor_map(&J.tmM, J.M, J.W, J.H, 4, S.ck.p_nb, br);
        if (!okm) {   // shape the TMA unit cannot describe: per-tile column pass
            S.p_cols = false;
            J.cpc = S.ck.nb < J.W ? S.ck.nb : J.W;
            J.n_col_tiles = (J.W + J.cpc - 1) / J.cpc;
        }
        J.use_tma_cols = S.p_cols ? 1 : 0;
        if (S.p_cols && S.ck.p_mt) J.Mt = (const float *)(a + S.oMt);
        S.p_half = S.p_cols && S.ck.p_col_split && encode_tensor_map(&J.tmXh, J.X, J.W, J.H, 8, S.ck.p_nb / 2, br);
    }
}

int job_modulus_tiles(const JobDev &J, cudaStream_t s)
{
    if (!J.Mt) return IMR_SUCCESS;
    const size_t n = (size_t)J.n_col_tiles * J.cpc * J.H;
    k_modulus_tiles<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(J.M, const_cast<float *>(J.Mt), J.W, J.H, J.cpc, n);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error("modulus tiles", e);
        return IMR_ERR_CUDA;
    }
    return IMR_SUCCESS;
}

int job_upload(const JobDev &J, const JobShape &S, char *a, JobDev *dj, cudaStream_t s)
{
    const size_t N = (size_t)J.W * J.H;
    CK(cudaMemcpyAsync(a + S.oW, S.wt.data(), S.wt.size() * 4, cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync(a + S.oT, S.taps.data(), S.taps.size() * 4, cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync(dj, &J, sizeof(JobDev), cudaMemcpyHostToDevice, s));
    CK(cudaMemsetAsync(a + S.oMask, 0, N, s));
    const size_t n_err = J.mode == kModeHio ? (size_t)J.n_err : (size_t)J.n_cycles + 1;   // allocated length
    CK(cudaMemsetAsync(a + S.oErr, 0, n_err * 4, s));
    return IMR_SUCCESS;
}
}  // namespace imr

extern "C" {

const char *imr_status_string(int s)
{
    switch (s) {
    case IMR_SUCCESS: return "success";
    case IMR_ERR_INVALID_VALUE: return "invalid value";
    case IMR_ERR_UNSUPPORTED_SIZE: return "unsupported image size";
    case IMR_ERR_OUT_OF_MEMORY: return "out of memory";
    case IMR_ERR_CUDA: return "CUDA error";
    case IMR_ERR_NOT_INITIALIZED: return "not initialised";
    case IMR_ERR_QUEUE: return "task queue error";
    case IMR_ERR_DEVICE_TIMEOUT: return "device-side wait timed out";
    case IMR_ERR_CANCELLED: return "cancelled";
    default: return "unknown status";
    }
}

const char *imr_last_error(void) { return g_last_error; }

unsigned imr_max_side(void) { return kMaxSide; }

int imr_side_supported(unsigned n) { return length_supported((int)n) ? 1 : 0; }

int imr_gaussian_weights(double sigma, float *h_w, int cap)
{
    if (!(sigma > 0)) return -1;
    return gaussian_weights(sigma, h_w, cap);
}

int imr_plan_destroy(imr_plan *P)
{
    if (!P) return IMR_SUCCESS;
    if (P->gexec) cudaGraphExecDestroy(P->gexec);
    if (P->graph) cudaGraphDestroy(P->graph);
    if (P->gexec_rem) cudaGraphExecDestroy(P->gexec_rem);
    if (P->graph_rem) cudaGraphDestroy(P->graph_rem);
    if (P->arena) cudaFree(P->arena);
    if (P->dbg_gprime) cudaFree(P->dbg_gprime);
    delete P;
    return IMR_SUCCESS;
}

// Capture the cycles as graphs: up to kPlanGraphCycles cycles per graph, so a
// reconstruction is one or a few graph launches (no host work between
// cycles), plus one graph for the remainder.  Replaces earlier graphs.
static int plan_capture(imr_plan *P)
{
    if (P->gexec) cudaGraphExecDestroy(P->gexec);
    if (P->graph) cudaGraphDestroy(P->graph);
    if (P->gexec_rem) cudaGraphExecDestroy(P->gexec_rem);
    if (P->graph_rem) cudaGraphDestroy(P->graph_rem);
    P->gexec = P->gexec_rem = nullptr;
    P->graph = P->graph_rem = nullptr;
    const JobDev &J = P->hj;
    P->chunk = J.n_cycles < kPlanGraphCycles ? J.n_cycles : kPlanGraphCycles;
    P->n_chunks = P->chunk ? J.n_cycles / P->chunk : 0;
    const int rem = P->chunk ? J.n_cycles % P->chunk : 0;
    int rc = IMR_SUCCESS;
    cudaStream_t cs;
    cudaError_t e = cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking);
    for (int g = 0; g < 2 && e == cudaSuccess && rc == IMR_SUCCESS; ++g) {
        const int cycles = g == 0 ? P->chunk : rem;
        if (cycles == 0) continue;
        cudaGraph_t &gr = g == 0 ? P->graph : P->graph_rem;
        cudaGraphExec_t &gx = g == 0 ? P->gexec : P->gexec_rem;
        e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
        if (e != cudaSuccess) break;
        for (int c = 0; c < cycles && rc == IMR_SUCCESS; ++c) rc = plan_launch_cycle(P, cs);
        cudaError_t e2 = cudaStreamEndCapture(cs, &gr);
        if (rc == IMR_SUCCESS && e2 == cudaSuccess)
            e = cudaGraphInstantiate(&gx, gr, 0);
        else if (e2 != cudaSuccess)
            e = e2;
    }
    cudaStreamDestroy(cs);
    if (e != cudaSuccess) {
        set_error("graph capture", e);
        return rc ? rc : IMR_ERR_CUDA;
    }
    return rc;
}

int imr_plan_create(imr_plan **out, unsigned W, unsigned H, const imr_params *params)
{
    if (!out || W == 0 || H == 0) return IMR_ERR_INVALID_VALUE;
    *out = nullptr;
    int rc = ensure_kernel_attributes();
    if (rc) return rc;
    imr_plan *P = new imr_plan();
    cudaGetDevice(&P->dev);
    P->W = (int)W;
    P->H = (int)H;
    resolve_params(params, P->p);
    JobDev &J = P->hj;
    JobShape S;
    if ((rc = job_prepare(W, H, P->p, J, S))) {
        delete P;
        return rc;
    }
    const size_t extra = (sizeof(JobState) + 255) / 256 * 256 + (sizeof(JobDev) + 255) / 256 * 256 +
                         (5 * sizeof(WorkList) + 255) / 256 * 256;
    cudaError_t e = device_alloc((void **)&P->arena, S.bytes + extra);
    if (e != cudaSuccess) {
        set_error("cudaMalloc plan arena", e);
        delete P;
        return IMR_ERR_OUT_OF_MEMORY;
    }
    char *a = (char *)P->arena;
    char *tail = a + S.bytes;
    JobState *st = (JobState *)tail;
    P->dj = (JobDev *)(tail + (sizeof(JobState) + 255) / 256 * 256);
    P->Lrow = (WorkList *)((char *)P->dj + (sizeof(JobDev) + 255) / 256 * 256);
    P->Lcol = P->Lrow + 1;
    P->Lvb = P->Lrow + 2;
    P->Lrow_n = P->Lrow + 3;
    P->Lcol_n = P->Lrow + 4;
    job_bind(J, S, a, st);
    P->st = J.st;
    P->rk = S.rk;
    P->ck = S.ck;
    P->p_rows = S.p_rows;
    P->p_cols = S.p_cols;
    P->smem_row = S.smem_row;
    P->smem_fin = S.smem_fin;
    P->smem_col = S.smem_col;
    if (P->p_rows) {
        P->g_row_first = persistent_grid((const void *)P->rk.p_hio_first, P->rk.threads, P->rk.p_smem_first,
                                         J.n_row_tiles);
        P->g_row = persistent_grid((const void *)P->rk.p_hio, P->rk.threads, P->rk.p_smem, J.n_row_tiles);
    }
    int n_split = 0;
    if (P->p_cols) {
        int g_max = persistent_grid((const void *)P->ck.p_col, P->ck.p_threads, P->ck.p_smem, 1 << 30);
        if (S.p_half && col_split(J.n_col_tiles, g_max)) {   // the half-tile variant of the pass
            P->ck.p_col = P->ck.p_col_split;
            g_max = persistent_grid((const void *)P->ck.p_col, P->ck.p_threads, P->ck.p_smem, 1 << 30);
            n_split = col_split(J.n_col_tiles, g_max);
        }
        P->g_col = std::min(g_max, J.n_col_tiles + n_split);
    }
    narrow_tiles(P->rk, P->ck, P->p_cols, P->W, P->H, &P->n_row_narrow, &P->n_col_narrow);
    P->dependent = passes_dependent(J, S, P->rk, P->ck, false, n_split, P->n_row_narrow > 0, P->n_col_narrow > 0);
    const bool one_item_cols = P->n_col_narrow || !P->p_cols;
    P->cols_dependent = P->dependent && (!P->n_row_narrow || !one_item_cols ||
                                         small_plan_columns_early(P->n_col_narrow ? P->n_col_narrow : J.n_col_tiles,
                                                                  P->n_col_narrow ? P->ck.n_threads : P->ck.threads));
    if (J.n_vb_tiles < 2 * 148) {   // tiles of 128 rows would leave SMs idle
        J.n_vb_tiles = J.vb_tiles_x * ((J.H + kVbTileYSmall - 1) / kVbTileYSmall);
        P->vblur = k_vblur<kVbTileYSmall>;
    }
    const WorkList lists[5] = {{nullptr, J.n_row_tiles, 0}, {nullptr, J.n_col_tiles, n_split}, {nullptr, J.n_vb_tiles, 0},
                               {nullptr, P->n_row_narrow, 0}, {nullptr, P->n_col_narrow, 0}};
    e = cudaMemcpy(P->Lrow, lists, sizeof(lists), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = job_upload(J, S, a, P->dj, 0) ? cudaErrorUnknown : cudaSuccess;
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e != cudaSuccess) {
        set_error("plan upload", e);
        imr_plan_destroy(P);
        return IMR_ERR_CUDA;
    }
    if ((rc = plan_capture(P))) {
        imr_plan_destroy(P);
        return rc;
    }
    *out = P;
    return IMR_SUCCESS;
}

int imr_plan_launches(imr_plan *P, long *launches)
{
    if (!P || !launches) return IMR_ERR_INVALID_VALUE;
    *launches = (P->hj.Mt && (!P->n_col_narrow || P->prec) ? 2 : 1) + (long)P->hj.n_cycles * (2 + 2L * P->hj.n_hio) + 2;
    return IMR_SUCCESS;
}

int imr_plan_execute(imr_plan *P, const float *d_modulus, float *d_out, void *stream)
{
    if (!P || !d_modulus || !d_out) return IMR_ERR_INVALID_VALUE;
    cudaStream_t s = (cudaStream_t)stream;
    const JobDev &J = P->hj;
    const size_t N = (size_t)P->W * P->H;
    CK(cudaMemcpyAsync((void *)J.M, d_modulus, N * 4, cudaMemcpyDeviceToDevice, s));
    if (!P->n_col_narrow || P->prec)   // the passes that read the modulus in tiles
        if (int rc = job_modulus_tiles(J, s)) return rc;
    CK(cudaMemsetAsync(P->st, 0, sizeof(JobState), s));
    P->ck.init<<<J.n_col_tiles, P->ck.threads, P->smem_col, s>>>(P->dj, P->Lcol);
    CK(cudaGetLastError());
    for (int c = 0; c < P->n_chunks; ++c) CK(cudaGraphLaunch(P->gexec, s));
    if (P->gexec_rem) CK(cudaGraphLaunch(P->gexec_rem, s));
    if (int rc = launch_finish(P->rk, J.n_row_tiles, P->smem_fin, s, P->dj, P->Lrow, P->dbg_gprime)) return rc;
    P->vblur<<<J.n_vb_tiles, kVbThreads, 0, s>>>(P->dj, P->Lvb);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(d_out, J.out, N * 4, cudaMemcpyDeviceToDevice, s));
    return IMR_SUCCESS;
}

int imr_plan_execute_host(imr_plan *P, const float *h_modulus, float *h_out, void *stream)
{
    if (!P || !h_modulus || !h_out) return IMR_ERR_INVALID_VALUE;
    cudaStream_t s = (cudaStream_t)stream;
    const JobDev &J = P->hj;
    const size_t N = (size_t)P->W * P->H;
    CK(cudaMemcpyAsync((void *)J.M, h_modulus, N * 4, cudaMemcpyHostToDevice, s));
    if (!P->n_col_narrow || P->prec)   // the passes that read the modulus in tiles
        if (int rc = job_modulus_tiles(J, s)) return rc;
    CK(cudaMemsetAsync(P->st, 0, sizeof(JobState), s));
    P->ck.init<<<J.n_col_tiles, P->ck.threads, P->smem_col, s>>>(P->dj, P->Lcol);
    CK(cudaGetLastError());
    for (int c = 0; c < P->n_chunks; ++c) CK(cudaGraphLaunch(P->gexec, s));
    if (P->gexec_rem) CK(cudaGraphLaunch(P->gexec_rem, s));
    if (int rc = launch_finish(P->rk, J.n_row_tiles, P->smem_fin, s, P->dj, P->Lrow, P->dbg_gprime)) return rc;
    P->vblur<<<J.n_vb_tiles, kVbThreads, 0, s>>>(P->dj, P->Lvb);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(h_out, J.out, N * 4, cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    return IMR_SUCCESS;
}

int imr_plan_stats(imr_plan *P, void *stream, int *cycles_done, float *errors)
{
    if (!P) return IMR_ERR_INVALID_VALUE;
    cudaStream_t s = (cudaStream_t)stream;
    CK(cudaStreamSynchronize(s));
    JobState st;
    CK(cudaMemcpy(&st, P->st, sizeof(JobState), cudaMemcpyDeviceToHost));
    if (cycles_done) *cycles_done = st.cycles_done;
    if (st.err) {
        snprintf(g_last_error, sizeof(g_last_error), "a device-side copy wait timed out");
        return IMR_ERR_DEVICE_TIMEOUT;
    }
    if (errors) CK(cudaMemcpy(errors, P->hj.errors, sizeof(float) * P->hj.n_cycles, cudaMemcpyDeviceToHost));
    return IMR_SUCCESS;
}

int imr_plan_copy_state(imr_plan *P, int what, void *h_dst, void *stream)
{
    if (!P || !h_dst) return IMR_ERR_INVALID_VALUE;
    cudaStream_t s = (cudaStream_t)stream;
    const size_t N = (size_t)P->W * P->H;
    const void *src = nullptr;
    size_t bytes = 0;
    switch (what) {
    case 0: src = P->hj.mask; bytes = N; break;
    case 1: src = P->hj.X; bytes = N * 8; break;
    case 2: src = P->hj.G; bytes = N * 8; break;
    case 3: src = P->hj.vb; bytes = N * 4; break;
    default: return IMR_ERR_INVALID_VALUE;
    }
    CK(cudaMemcpyAsync(h_dst, src, bytes, cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    return IMR_SUCCESS;
}

// One replay of `iters` (row pass, column pass) pairs captured into a graph;
// with `split`, an event record node after every pass (ev[0..2*iters]),
// else only before and after the pairs (ev[0], ev[1]).  External records: a
// plain record inside a capture only orders streams.
static cudaError_t profile_replay(imr_plan *P, int iters, bool split, cudaStream_t s, std::vector<cudaEvent_t> &ev)
{
    cudaStream_t cs = nullptr;
    cudaError_t e = cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking);
    if (e != cudaSuccess) return e;
    cudaGraph_t gr = nullptr;
    cudaGraphExec_t gx = nullptr;
    e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
        int k = 0;
        cudaEventRecordWithFlags(ev[k++], cs, cudaEventRecordExternal);
        for (int i = 0; i < iters; ++i) {
            if (e == cudaSuccess) e = plan_launch_row(P, false, cs);
            if (split) cudaEventRecordWithFlags(ev[k++], cs, cudaEventRecordExternal);
            if (e == cudaSuccess) e = plan_launch_col(P, cs);
            if (split || i == iters - 1) cudaEventRecordWithFlags(ev[k++], cs, cudaEventRecordExternal);
        }
        const cudaError_t e2 = cudaStreamEndCapture(cs, &gr);
        if (e == cudaSuccess) e = e2 != cudaSuccess ? e2 : cudaGraphInstantiate(&gx, gr, 0);
    }
    if (e == cudaSuccess) e = cudaMemsetAsync(P->st, 0, sizeof(JobState), s);
    if (e == cudaSuccess) e = cudaGraphLaunch(gx, s);   // warm-up
    if (e == cudaSuccess) e = cudaGraphLaunch(gx, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (gx) cudaGraphExecDestroy(gx);
    if (gr) cudaGraphDestroy(gr);
    cudaStreamDestroy(cs);
    return e;
}

int imr_plan_profile(imr_plan *P, int iters, void *stream, float *ms_row, float *ms_col)
{
    if (!P || iters < 1 || !ms_row || !ms_col) return IMR_ERR_INVALID_VALUE;
    cudaStream_t s = (cudaStream_t)stream;
    // The pair time comes from a graph of `iters` pairs with no event inside
    // (kernel after kernel, as a reconstruction runs them: an event between
    // two kernels drains the GPU and adds that gap to the pass); its split
    // between the two passes from a replay with an event after every pass.
    std::vector<cudaEvent_t> ev(2 * iters + 1, nullptr);
    for (auto &x : ev) CK(cudaEventCreate(&x));
    cudaError_t e = profile_replay(P, iters, false, s, ev);
    float pair = 0;
    if (e == cudaSuccess) e = cudaEventElapsedTime(&pair, ev[0], ev[1]);
    if (e == cudaSuccess) e = profile_replay(P, iters, true, s, ev);
    double tr = 0, tc = 0;
    for (int i = 0; i < iters && e == cudaSuccess; ++i) {
        float a = 0, b = 0;
        e = cudaEventElapsedTime(&a, ev[2 * i], ev[2 * i + 1]);
        if (e == cudaSuccess) e = cudaEventElapsedTime(&b, ev[2 * i + 1], ev[2 * i + 2]);
        tr += a;
        tc += b;
    }
    for (auto &x : ev) cudaEventDestroy(x);
    if (e != cudaSuccess) {
        set_error("imr_plan_profile", e);
        return IMR_ERR_CUDA;
    }
    const double per_pair = (double)pair / iters, frac_row = tr + tc > 0 ? tr / (tr + tc) : 0.5;
    *ms_row = (float)(per_pair * frac_row);
    *ms_col = (float)(per_pair * (1.0 - frac_row));
    return IMR_SUCCESS;
}

int imr_plan_pass_bytes(imr_plan *P, double *row_bytes, double *col_bytes)
{
    if (!P || !row_bytes || !col_bytes) return IMR_ERR_INVALID_VALUE;
    const double N = (double)P->W * P->H;
    *row_bytes = 33.0 * N;
    *col_bytes = 20.0 * N;
    return IMR_SUCCESS;
}

int imr_plan_set_wait_limit(imr_plan *P, unsigned long long limit_ns)
{
    if (!P) return IMR_ERR_INVALID_VALUE;
    P->hj.wait_ns = limit_ns;
    // the captured graphs read the job description from device memory: no re-capture
    CK(cudaMemcpy(P->dj, &P->hj, sizeof(JobDev), cudaMemcpyHostToDevice));
    return IMR_SUCCESS;
}

int imr_plan_set_precision(imr_plan *P, int precision)
{
    if (!P || precision < IMR_PREC_FP32 || precision > IMR_PREC_FP16X3) return IMR_ERR_INVALID_VALUE;
    if (precision != IMR_PREC_FP32 && !(P->p_cols && P->ck.p_col_tc[precision - 1])) {
        snprintf(g_last_error, sizeof(g_last_error),
                 "split-precision column pass: height %d is not a power of two in 256..4096 with a pipelined "
                 "column pass", P->H);
        return IMR_ERR_UNSUPPORTED_SIZE;
    }
    if (precision == P->prec) return IMR_SUCCESS;
    P->prec = precision;
    if (precision != IMR_PREC_FP32)
        P->g_col_tc = persistent_grid((const void *)P->ck.p_col_tc[precision - 1], P->ck.p_threads, P->ck.p_smem_tc,
                                      P->hj.n_col_tiles);
    CK(cudaDeviceSynchronize());
    return plan_capture(P);
}

int imr_fft2d_split(void *d_data, unsigned W, unsigned H, int sign, int precision, void *stream)
{
    if (!d_data || W == 0 || H == 0 || (sign != 1 && sign != -1) || precision < IMR_PREC_BF16X3 ||
        precision > IMR_PREC_FP16X3)
        return IMR_ERR_INVALID_VALUE;
    int rc = ensure_kernel_attributes();
    if (rc) return rc;
    const ColKernels ck = col_kernels((int)H);
    auto kcol = ck.fft_tc[precision - 1][sign < 0 ? 0 : 1];
    if (!kcol || W % (unsigned)ck.p_nb != 0 || ((uintptr_t)d_data & 15)) {
        snprintf(g_last_error, sizeof(g_last_error),
                 "imr_fft2d_split: H must be a power of two in 256..4096 and W a multiple of %d", ck.p_nb);
        return IMR_ERR_UNSUPPORTED_SIZE;
    }
    FftPlanDev pr, pc;
    if ((rc = make_fft_plan((int)W, pr)) || (rc = make_fft_plan((int)H, pc))) return rc;
    JobDev J;
    memset(&J, 0, sizeof(J));
    J.W = (int)W;
    J.H = (int)H;
    J.X = (float2 *)d_data;
    J.pcol = pc;
    J.cpc = ck.p_nb;
    J.n_col_tiles = (int)W / ck.p_nb;
    if (!encode_tensor_map(&J.tmX, d_data, J.W, J.H, 8, ck.p_nb, ck.p_box_rows)) return IMR_ERR_UNSUPPORTED_SIZE;
    cudaStream_t s = (cudaStream_t)stream;
    char *dev = nullptr;
    const size_t jb = (sizeof(JobDev) + 255) / 256 * 256;
    CK(scratch_alloc((void **)&dev, jb + 256 + 256, s));
    JobDev *dj = (JobDev *)dev;
    WorkList *dl = (WorkList *)(dev + jb);
    JobState *dst = (JobState *)(dev + jb + 256);
    J.st = dst;
    const WorkList wl{nullptr, J.n_col_tiles};
    CK(cudaMemcpyAsync(dj, &J, sizeof(JobDev), cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync(dl, &wl, sizeof(WorkList), cudaMemcpyHostToDevice, s));
    CK(cudaMemsetAsync(dst, 0, sizeof(JobState), s));
    const int grid = persistent_grid((const void *)kcol, ck.p_threads, ck.p_smem_tc, J.n_col_tiles);
    if (sign < 0) {
        if ((rc = fft_passes((float2 *)d_data, (int)W, (int)H, -1, 1, pr, pc, s))) return rc;
        kcol<<<grid, ck.p_threads, ck.p_smem_tc, s>>>(dj, dl);
    } else {
        kcol<<<grid, ck.p_threads, ck.p_smem_tc, s>>>(dj, dl);
        if ((rc = fft_passes((float2 *)d_data, (int)W, (int)H, +1, 1, pr, pc, s))) return rc;
    }
    CK(cudaGetLastError());
    JobState st;
    CK(cudaMemcpyAsync(&st, dst, sizeof(JobState), cudaMemcpyDeviceToHost, s));
    CK(cudaFreeAsync(dev, s));
    CK(cudaStreamSynchronize(s));
    if (st.err) {
        snprintf(g_last_error, sizeof(g_last_error), "imr_fft2d_split: a device-side copy wait timed out");
        return IMR_ERR_DEVICE_TIMEOUT;
    }
    return IMR_SUCCESS;
}

int imr_bounded_wait_check(unsigned long long limit_ns, unsigned long long *elapsed_ns, void *stream)
{
    cudaStream_t s = (cudaStream_t)stream;
    k_wait_probe<<<1, 32, 0, s>>>(limit_ns);
    CK(cudaGetLastError());
    unsigned long long r[2] = {0, 0};
    CK(cudaMemcpyFromSymbolAsync(r, g_wait_probe, sizeof(r), 0, cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    if (elapsed_ns) *elapsed_ns = r[1];
    if (r[0] == 0) {
        snprintf(g_last_error, sizeof(g_last_error), "bounded wait gave up after %llu ns", r[1]);
        return IMR_ERR_DEVICE_TIMEOUT;
    }
    return IMR_SUCCESS;
}

// ------------------------------------------------------------ drop-in
int imr_cuda_shrink_wrap(float *io, unsigned W, unsigned H, void *stream, unsigned nBlocks,
                         unsigned nThreads, unsigned nCycles, float targetError, float hioBeta,
                         float cutAuto, float cut, float sigma0, float sigmaChange,
                         unsigned nHio)
{
    (void)nBlocks;
    (void)nThreads;
    if (!io || W == 0 || H == 0) return IMR_ERR_INVALID_VALUE;
    imr_params p{nCycles, targetError, hioBeta, cutAuto, cut, sigma0, sigmaChange, nHio};
    imr_plan *P = nullptr;
    int rc = plan_cache_acquire(W, H, &p, &P);
    if (rc) return rc;
    rc = imr_plan_execute_host(P, io, io, stream);
    plan_cache_release(P);
    return rc;
}

// ------------------------------------------------------------ kernel-level
int imr_fft2d(void *d_data, unsigned W, unsigned H, int sign, void *stream)
{
    if (!d_data || W == 0 || H == 0 || (sign != 1 && sign != -1)) return IMR_ERR_INVALID_VALUE;
    int dev = 0;
    CK(cudaGetDevice(&dev));
    // the plans and kernels of the thread's last size (their tables live as long
    // as the process)
    static thread_local struct {
        int dev = -1;
        unsigned W = 0, H = 0;
        FftPlanDev pr, pc;
        RowKernels rk;
        ColKernels ck;
    } last;
    if (last.dev != dev || last.W != W || last.H != H) {
        last.dev = -1;
        int rc = ensure_kernel_attributes();
        if (rc) return rc;
        if ((rc = make_fft_plan((int)W, last.pr)) || (rc = make_fft_plan((int)H, last.pc))) return rc;
        last.rk = row_kernels((int)W);
        last.ck = col_kernels((int)H, (int)W);
        last.W = W;
        last.H = H;
        last.dev = dev;
    }
    return fft_launch((float2 *)d_data, (int)W, (int)H, sign, 3, last.pr, last.pc, last.rk, last.ck,
                      (cudaStream_t)stream);
}

int imr_gaussian_blur(float *d_data, float *d_tmp, unsigned W, unsigned H, double sigma, int axes,
                      void *stream)
{
    if (!d_data || W == 0 || H == 0 || !(sigma > 0) || axes < 1 || axes > 3) return IMR_ERR_INVALID_VALUE;
    if ((axes & 2) && !d_tmp) return IMR_ERR_INVALID_VALUE;
    if (W > 65536 || H > 65536) return IMR_ERR_UNSUPPORTED_SIZE;
    int rc = ensure_kernel_attributes();
    if (rc) return rc;
    Taps t;
    memset(&t, 0, sizeof(t));
    const int K = gaussian_weights(sigma, t.w, kMaxTaps);
    if (K > kMaxTaps) return IMR_ERR_INVALID_VALUE;
    cudaStream_t s = (cudaStream_t)stream;
    // both axes: rows into the scratch image, columns back from it
    float *const rows_out = axes == 3 ? d_tmp : d_data;
    if (axes & 1) {
        const bool vec = W % 4 == 0 && (((uintptr_t)d_data | (uintptr_t)rows_out) & 15) == 0;
        if (hblur_rolling((int)W, (int)H, K, vec)) {
            const int rs = hb_row_floats((int)W), chunks = rs / kHbOut, pw = (int)W / (vec ? 4 : 1);
            const int nr = std::max(1, std::min(kRowThreads / chunks, (int)H / 296));
            const int threads = std::max(nr == 1 ? 32 : vec ? 128 : kRowThreads,
                                         std::min(kRowThreads, (nr * chunks + 31) / 32 * 32));
            int lgx = 0;   // 2^lgx threads a row
            while ((1 << lgx) < pw) ++lgx;
            if ((1 << lgx) > threads) lgx = -1;
            const size_t rows_bytes = (size_t)nr * rs * 4;
            const bool staged = chunks > kRowThreads && rows_bytes + kHbStage * 4 + kTapStride * 4 <= (size_t)g_optin_smem;
            (vec ? k_hblur<true> : k_hblur<false>)<<<(H + nr - 1) / nr, threads, rows_bytes + (staged ? kHbStage * 4 : 0),
                                                     s>>>(d_data, rows_out, (int)W, (int)H, nr, lgx, staged, t, K);
        } else {
            k_hblur_px<<<H, kRowThreads, (size_t)W * 4, s>>>(d_data, rows_out, (int)W, t, K);
        }
    }
    if (axes & 2) {
        const int tx = (int)((W + kVbTileX - 1) / kVbTileX), nt = tx * (int)((H + kVbTileY - 1) / kVbTileY);
        const float *const in = axes == 3 ? d_tmp : d_data;
        float *const out = axes == 3 ? d_data : d_tmp;
        if (!vblur_small_tiles(nt))
            k_vblur_plain<kVbTileY><<<nt, kVbThreads, 0, s>>>(in, out, (int)W, (int)H, t, K, nullptr);
        else
            k_vblur_plain<kVbTileYSmall><<<tx * (int)((H + kVbTileYSmall - 1) / kVbTileYSmall), kVbThreads, 0, s>>>(
                in, out, (int)W, (int)H, t, K, nullptr);
        if (axes == 2) CK(cudaMemcpyAsync(d_data, d_tmp, (size_t)W * H * 4, cudaMemcpyDeviceToDevice, s));
    }
    CK(cudaGetLastError());
    return IMR_SUCCESS;
}

int imr_diffraction_intensity(float *h_io, unsigned W, unsigned H, void *stream)
{
    if (!h_io || W == 0 || H == 0) return IMR_ERR_INVALID_VALUE;
    if (!length_supported((int)W) || !length_supported((int)H)) return IMR_ERR_UNSUPPORTED_SIZE;
    cudaStream_t s = (cudaStream_t)stream;
    const size_t N = (size_t)W * H;
    char *buf = nullptr;
    CK(scratch_alloc((void **)&buf, N * 12, s));
    float2 *d = (float2 *)buf;
    float *f = (float *)(buf + N * 8);
    const int g = (int)std::min<size_t>((N + 255) / 256, 148 * 16);
    cudaError_t e = cudaMemcpyAsync(f, h_io, N * 4, cudaMemcpyHostToDevice, s);
    int rc = IMR_SUCCESS;
    if (e == cudaSuccess) {
        k_real_to_complex<<<g, 256, 0, s>>>(f, d, (long)N);
        rc = imr_fft2d(d, W, H, -1, stream);
    }
    if (e == cudaSuccess && rc == IMR_SUCCESS) {
        k_complex_norm<<<g, 256, 0, s>>>(d, f, (long)N);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpyAsync(h_io, f, N * 4, cudaMemcpyDeviceToHost, s);
    }
    cudaFreeAsync(buf, s);
    if (rc) return rc;
    CK(e);
    CK(cudaStreamSynchronize(s));
    return IMR_SUCCESS;
}

int imr_release_scratch(void)
{
    CK(scratch_release());
    return IMR_SUCCESS;
}

int imr_vector_max(const float *d, size_t n, float *h_max, void *stream)
{
    if (!d || !h_max) return IMR_ERR_INVALID_VALUE;
    if (n == 0) {
        *h_max = -FLT_MAX;
        return IMR_SUCCESS;
    }
    cudaStream_t s = (cudaStream_t)stream;
    unsigned *dk = nullptr;
    CK(scratch_alloc((void **)&dk, sizeof(unsigned), s));
    CK(cudaMemsetAsync(dk, 0, sizeof(unsigned), s));
    long blocks = (long)((n + 255) / 256);
    if (blocks > 148 * 8) blocks = 148 * 8;
    k_vector_max<<<(unsigned)blocks, 256, 0, s>>>(d, (long)n, dk);
    CK(cudaGetLastError());
    unsigned key = 0;
    CK(cudaMemcpyAsync(&key, dk, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
    CK(cudaFreeAsync(dk, s));
    CK(cudaStreamSynchronize(s));
    unsigned u = (key & 0x80000000u) ? (key & 0x7fffffffu) : ~key;
    memcpy(h_max, &u, 4);
    return IMR_SUCCESS;
}

}  // extern "C"

// ------------------------------------------------------------ plan cache
// Idle plans keyed by (device, W, H, parameters), so repeated drop-in calls
// of one size reuse buffers and the captured graph.  Concurrent callers of
// the same size get separate plans.
namespace imr {
struct PlanKey {
    int dev;
    unsigned W, H;
    imr_params p;
    bool operator<(const PlanKey &o) const { return memcmp(this, &o, sizeof(PlanKey)) < 0; }
};
static std::mutex g_cache_mu;
static std::multimap<PlanKey, imr_plan *> g_idle;

int plan_cache_acquire(unsigned W, unsigned H, const imr_params *params, imr_plan **out)
{
    PlanKey k;
    memset(&k, 0, sizeof(k));
    cudaGetDevice(&k.dev);
    k.W = W;
    k.H = H;
    resolve_params(params, k.p);
    {
        std::lock_guard<std::mutex> lk(g_cache_mu);
        auto it = g_idle.find(k);
        if (it != g_idle.end()) {
            *out = it->second;
            g_idle.erase(it);
            return IMR_SUCCESS;
        }
    }
    return imr_plan_create(out, W, H, &k.p);
}

void plan_cache_release(imr_plan *P)
{
    PlanKey k;
    memset(&k, 0, sizeof(k));
    k.dev = P->dev;
    k.W = (unsigned)P->W;
    k.H = (unsigned)P->H;
    k.p = P->p;
    std::lock_guard<std::mutex> lk(g_cache_mu);
    g_idle.insert(std::make_pair(k, P));
}
}  // namespace imr
