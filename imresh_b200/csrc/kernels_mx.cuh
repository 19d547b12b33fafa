// Passes for lengths 2^a 3^b 5^c 7^d that have no compile-time kernel.
//
// The transform is fft_dev.cuh's Stockham schedule of the length (FftPlanDev::rad:
// 8s, then 4 / 2, 3s, 5s, 7s; one table twiddle per value and pass), with the
// same operations on every value, so its results are the schedule's bit for
// bit.  What differs is how the passes run: two consecutive radices R1, R2
// whose product is at most 16 run as one grouped pass on registers.
// With L = n/(R1 R2) and k = j mod Ns, thread j < L
//     loads   x[j + s L], s = q1 R2 + q2,
//     runs the R2 butterflies of radix R1 (twiddle q1 k n/(Ns R1)) and the
//     R1 butterflies of radix R2 (twiddle q2 (k + q1 Ns) n/(Ns R1 R2)),
//     stores  y[(j - k) R1 R2 + k + q1 Ns + q2 Ns R1],
// so 600 = 8 (3 5) 5 makes two shared-memory exchanges instead of three.
//
// What bounds these passes: at the sizes that run here (a few hundred to 2048
// a side) a pass is a chain of latencies -- global load, one exchange per
// grouped pass, store -- and of instruction fetch (a short kernel runs cold
// code), not bandwidth.  The form they replace held every butterfly of a thread
// in registers across two barriers per radix (255 registers, one 8-warp CTA
// per SM), divided by run-time lengths for every butterfly, and loaded g_prev
// and the mask one element after another.  Here passes ping-pong between two
// buffers (one barrier each, no values live across it), the divisions are
// multiplications by host-made reciprocals, the operands are requested together
// with X, and the twiddle table is in shared memory beside them.  Measured per
// HIO iteration (row + column pass), before -> now: 100 x 100 24.2 -> 10.0 us,
// 600 x 300 34.6 -> 16.6, 1000 x 800 111 -> 34.7, 1920 x 1080 328 -> 75.
// Radix pairs up to 25 (8 3, 5 5, ...) on half the blocks per SM made fewer
// exchanges but longer chains: 600 x 300 26 us, 1000 x 800 41, 1920 x 1080 89.
#pragma once

namespace imr {

constexpr int kMxRowThreads = 256;
constexpr int kMxRowElems = 2048;     // values of a row tile at most
constexpr int kMxColW = 4;            // columns of a column tile: 32-byte sectors
constexpr int kMxColWFew = 2;         // the same for few long columns (mx_few_columns)
// Blocks of a column pass per SM: few columns are no more than one.
__host__ __device__ constexpr int mx_col_blocks(int T, int C) { return C == kMxColWFew ? 1 : T == 256 ? 3 : 2; }
// Threads of a column tile: one butterfly of a grouped pass each, about (4 n / 16).
__host__ __device__ constexpr int mx_col_threads(int n) { return n > 1024 ? 512 : 256; }

// ---- shared-memory indices -----------------------------------------------------
// Rows are flat (sequence b at b*n): one spare value per 32; column tiles hold
// element e of column c at (e ^ ((e >> 4) & 15))*C + c.  Of the paddings
// and swizzles tried over all passes of all lengths in a model of the banks these
// needed the fewest wavefronts that one layout for every length gets: 1.36 and
// 1.24 of a conflict-free exchange (none: 1.63 and 1.33).
__host__ __device__ constexpr int mx_row_pad(int n) { return n + (n >> 5) + 1; }
template <int C>
__host__ __device__ constexpr int mx_col_pad(int n) { return ((n + 15) & ~15) * C; }
__device__ __forceinline__ int mx_row_at(int f) { return f + (f >> 5); }
template <int C>
__device__ __forceinline__ int mx_col_at(int e, int c) { return (e ^ ((e >> 4) & 15)) * C + c; }

// bytes: two exchange buffers, one operand per value (g_prev rows / modulus
// column tile), the twiddle table
__host__ __device__ constexpr int mx_row_smem(int n, int nb) { return (2 * mx_row_pad(nb * n) + nb * n + n) * 8; }
template <int C>
__host__ __device__ constexpr int mx_col_smem(int n)
{
    return 2 * mx_col_pad<C>(n) * 8 + mx_col_pad<C>(n) * 4 + n * 8;
}

// z *= w, the twiddle step.  The schedule's rounding, pinned: forward
// re = fma(zx, wx, -(zy wy)), im = fma(zx, wy, zy wx); an inverse transform,
// which runs here on conjugates (see mx_fft), fuses the other product of im.
__device__ __forceinline__ float2 mx_cmul_fwd(float2 z, float2 w)
{
    return make_float2(__fmaf_rn(z.x, w.x, -__fmul_rn(z.y, w.y)), __fmaf_rn(z.x, w.y, __fmul_rn(z.y, w.x)));
}
__device__ __forceinline__ float2 mx_cmul_inv(float2 z, float2 w)
{
    return make_float2(__fmaf_rn(z.x, w.x, -__fmul_rn(z.y, w.y)), __fmaf_rn(z.y, w.x, __fmul_rn(z.x, w.y)));
}

// ---- one grouped pass ------------------------------------------------------------
// C > 0: column tile of C sequences, else nseq flat rows.  T threads.
template <int R1, int R2, int C, int T>
__device__ __forceinline__ void mx_pass(const float2 *src, float2 *dst, const float2 *tw, const FftPass &P, int n,
                                        int nseq, bool inv)
{
    constexpr int R = R1 * R2;
    const int L = P.L, Ns = P.Ns;
    const int st1 = P.st1, st2 = P.st2;
    const int total = C ? C * L : nseq * L;
    for (int u = threadIdx.x; u < total; u += T) {
        int b, j;
        if constexpr (C > 0) {
            b = u % C;
            j = u / C;
        } else {
            b = P.mL ? (int)__umulhi((unsigned)u, P.mL) : u;   // u / L
            j = u - b * L;
        }
        const int k = P.mNs ? j - (int)__umulhi((unsigned)j, P.mNs) * Ns : 0;   // j mod Ns
        float2 v[R];
#pragma unroll
        for (int s = 0; s < R; ++s) v[s] = src[C ? mx_col_at<C>(j + s * L, b) : mx_row_at(b * n + j + s * L)];
        if (k != 0) {
            float2 w[R1];
#pragma unroll
            for (int q1 = 1; q1 < R1; ++q1) w[q1] = tw[q1 * k * st1];
            if (!inv) {
#pragma unroll
                for (int s = R2; s < R; ++s) v[s] = mx_cmul_fwd(v[s], w[s / R2]);
            } else {
#pragma unroll
                for (int s = R2; s < R; ++s) v[s] = mx_cmul_inv(v[s], w[s / R2]);
            }
        }
#pragma unroll
        for (int q2 = 0; q2 < R2; ++q2) {
            float2 a[R1];
#pragma unroll
            for (int q1 = 0; q1 < R1; ++q1) a[q1] = v[q1 * R2 + q2];
            dftR<R1, -1>(a);
#pragma unroll
            for (int q1 = 0; q1 < R1; ++q1) v[q1 * R2 + q2] = a[q1];
        }
        if constexpr (R2 > 1) {
#pragma unroll
            for (int q1 = 0; q1 < R1; ++q1) {
                const int k2 = k + q1 * Ns;
                float2 a[R2];
#pragma unroll
                for (int q2 = 0; q2 < R2; ++q2) a[q2] = v[q1 * R2 + q2];
                if (q1 > 0 || k != 0) {
                    float2 w[R2];
#pragma unroll
                    for (int q2 = 1; q2 < R2; ++q2) w[q2] = tw[q2 * k2 * st2];
                    if (!inv) {
#pragma unroll
                        for (int q2 = 1; q2 < R2; ++q2) a[q2] = mx_cmul_fwd(a[q2], w[q2]);
                    } else {
#pragma unroll
                        for (int q2 = 1; q2 < R2; ++q2) a[q2] = mx_cmul_inv(a[q2], w[q2]);
                    }
                }
                dftR<R2, -1>(a);
#pragma unroll
                for (int q2 = 0; q2 < R2; ++q2) v[q1 * R2 + q2] = a[q2];
            }
        }
        const int o = (j - k) * R + k;
#pragma unroll
        for (int q1 = 0; q1 < R1; ++q1)
#pragma unroll
            for (int q2 = 0; q2 < R2; ++q2) {
                const int e = o + (q1 + q2 * R1) * Ns;
                dst[C ? mx_col_at<C>(e, b) : mx_row_at(b * n + e)] = v[q1 * R2 + q2];
            }
    }
}

// Transform of the sequences in the buffer at offset a of the dynamic shared
// memory (b: the other buffer's offset); returns the offset of the buffer that
// holds the result.  Offsets, not pointers: selected between two buffers, a
// pointer becomes a generic one, and a pass through generic loads took twice
// as long.  The caller's writes of a are followed by a barrier; ends with a
// barrier (with no passes, n = 1, it does nothing).
//
// An inverse transform (inv) is the conjugate of the forward transform of the
// conjugate; the callers conjugate on the way in and out.  Apart from the
// twiddle step's choice of the fused product, every operation of the schedule
// commutes with negating the imaginary parts, so the values are the inverse
// schedule's (up to the sign of a zero).  The passes of an iteration run both transforms through this one
// body, in a loop: a kernel is short and its code cold, and with a second copy
// of the passes the second transform took twice the first one's time (7400
// cycles after 3700 for a row of 600, waiting for instructions).
template <int C, int T>
__device__ __forceinline__ int mx_fft(int a, int b, int otw, const FftPlanDev &p, int nseq, bool inv)
{
    extern __shared__ float4 smem4[];
    float2 *const sm = reinterpret_cast<float2 *>(smem4);
    const int n = p.n, npass = p.npass;
    for (int i = 0; i < npass; ++i) {
        const FftPass P = p.pass[i];
        switch (P.r1 * 16 + P.r2) {
#define MXP(R1, R2)                                                                \
    case (R1) * 16 + (R2):                                                         \
        mx_pass<R1, R2, C, T>(sm + a, sm + b, sm + otw, P, n, nseq, inv);     \
        break;
            MXP(8, 2) MXP(8, 1)
            MXP(4, 4) MXP(4, 3) MXP(4, 1)
            MXP(2, 7) MXP(2, 5) MXP(2, 3) MXP(2, 1)
            MXP(3, 5) MXP(3, 3) MXP(3, 1)
            MXP(5, 1) MXP(7, 1)
#undef MXP
        default: break;
        }
        __syncthreads();
        const int t = a;
        a = b;
        b = t;
    }
    return a;
}

// The plan of a length as words, one per thread, to be stored to shared memory
// with mx_store_plan (the passes read it all the time).
constexpr int kMxPlanWords = sizeof(FftPlanDev) / 4;
static_assert(sizeof(FftPlanDev) % 4 == 0 && kMxPlanWords <= 256, "plan copied as one word per thread");
__device__ __forceinline__ int mx_plan_word(const FftPlanDev &g)
{
    return threadIdx.x < kMxPlanWords ? reinterpret_cast<const int *>(&g)[threadIdx.x] : 0;
}
__device__ __forceinline__ void mx_store_plan(FftPlanDev *sp, int word)
{
    if (threadIdx.x < kMxPlanWords) reinterpret_cast<int *>(sp)[threadIdx.x] = word;
}

// ---- rows ---------------------------------------------------------------------
// row pass (see b_row_hio).  Everything a tile needs is requested before
// anything is waited for: the job's fields, then X, g_prev, the mask, the
// table and the state (g_prev of the first iteration, not yet written, is read
// and not used).
template <bool FIRST, bool FIX>
__global__ void __launch_bounds__(kMxRowThreads, 3) k_row_hio_mx(const JobDev *jobs, const WorkList *L)
{
    extern __shared__ float4 smem4[];
    float2 *const sm = reinterpret_cast<float2 *>(smem4);
    __shared__ FftPlanDev sp;
    constexpr int T = kMxRowThreads, V = kMxRowElems / T;
    const WorkList l = list_and_job0(jobs, L);
    int job = -1;
    for (int it = blockIdx.x; it < l.n; it += gridDim.x) {
        const WorkItem wi = l.items ? l.items[it] : WorkItem{0, it};
        const JobDev &J = jobs[wi.job];
        JobState *const st = J.st;
        const int W = J.W, rpc = J.rpc, y0 = wi.tile * rpc, nr = min(rpc, J.H - y0), n = nr * W;
        const size_t base = (size_t)y0 * W;
        float2 *const X = J.X + base, *const G = J.G + base;
        uint8_t *const mask = J.mask + base;
        const float2 *const gtw = J.prow.tw;
        const float beta = J.beta;
        const bool other = job != wi.job;   // (after the barrier that ended the last item)
        const int word = other ? mx_plan_word(J.prow) : 0;
        if (job < 0) pdl_wait();
        const int oa = 0, ob = mx_row_pad(rpc * W), og = 2 * ob, ot = og + rpc * W;
        float2 xv[V];
#pragma unroll
        for (int m = 0; m < V; ++m) {
            const int i = threadIdx.x + m * T;
            if (i < n) xv[m] = X[i];
        }
#pragma unroll
        for (int m = 0; m < V; ++m) {
            const int i = threadIdx.x + m * T;
            if (i < n) cp_async8(sm + og + i, G + i);
        }
        if (other)
            for (int i = threadIdx.x; i < W; i += T) cp_async8(sm + ot + i, gtw + i);
        uint8_t mk[V];
#pragma unroll
        for (int m = 0; m < V; ++m) {
            const int i = threadIdx.x + m * T;
            mk[m] = !FIRST && i < n ? mask[i] : 0;
        }
        const int stop = st->stop;
        const float thr = FIRST ? st->thr : 0.f;
        const int k = FIX ? st->cycle : FIRST ? st->hio_cycle : 1;
        const bool init_gprev = k == 0;
        const bool fin = FIX && k >= J.n_cycles;
        const bool track = FIX && (J.target > 0.f || fin);
        if (other) mx_store_plan(&sp, word);
        job = wi.job;
#pragma unroll
        for (int m = 0; m < V; ++m) {   // conjugated: the first transform is the inverse one
            const int i = threadIdx.x + m * T;
            if (i < n) sm[oa + mx_row_at(i)] = make_float2(xv[m].x, -xv[m].y);
        }
        cp_async_wait();
        __syncthreads();
        if (stop) continue;
        int r = oa;
        double tot = 0.0;
        unsigned cnt = 0u;
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
            r = mx_fft<0, T>(r, oa + ob - r, ot, sp, nr, h == 0);
            if (h == 1) break;
            if (it + (int)gridDim.x >= l.n) pdl_trigger();
            if (FIRST) {
                const float *const vb = J.vb + base;
                float bl[V];
#pragma unroll
                for (int m = 0; m < V; ++m) {
                    const int i = threadIdx.x + m * T;
                    bl[m] = i < n ? vb[i] : 0.f;
                }
#pragma unroll
                for (int m = 0; m < V; ++m) {
                    const int i = threadIdx.x + m * T;
                    mk[m] = bl[m] < thr ? 1 : 0;
                    if (i < n) mask[i] = mk[m];
                }
            }
#pragma unroll
            for (int m = 0; m < V; ++m) {
                const int i = threadIdx.x + m * T;
                if (i >= n) continue;
                float2 gp1 = sm[r + mx_row_at(i)];   // g'
                gp1.y = -gp1.y;
                if (FIX) {
                    if (track) hio_track(J.out, base + i, gp1, mk[m], tot, cnt);
                    if (fin) continue;
                }
                const float2 gp = init_gprev ? gp1 : sm[og + i];
                float2 g;
                if ((FIX ? mk[m] == 1 : mk[m] != 0) || gp1.x < 0.f)
                    g = make_float2(__fsub_rn(gp.x, __fmul_rn(beta, gp1.x)), __fsub_rn(gp.y, __fmul_rn(beta, gp1.y)));
                else
                    g = gp1;
                G[i] = g;
                sm[r + mx_row_at(i)] = g;
            }
            if (fin) break;
            __syncthreads();
        }
        if (!fin) {
#pragma unroll
            for (int m = 0; m < V; ++m) {
                const int i = threadIdx.x + m * T;
                if (i < n) X[i] = sm[r + mx_row_at(i)];
            }
        }
        if (FIX) hio_tile_done<T>(J, wi.tile, tot, cnt, J.n_row_tiles);
        __syncthreads();
    }
}

// once per cycle (see b_row_finish); a template so that only the translation
// unit that launches it compiles it
template <int>
__global__ void __launch_bounds__(kMxRowThreads, 3) k_row_finish_mx(const JobDev *jobs, const WorkList *L,
                                                                  float2 *dbg_gprime)
{
    extern __shared__ float4 smem4[];
    float2 *const sm = reinterpret_cast<float2 *>(smem4);
    __shared__ FftPlanDev sp;
    __shared__ float wsm[kTapStride];
    constexpr int T = kMxRowThreads, V = kMxRowElems / T;
    __shared__ double red[2 * T / 32];
    const WorkList l = list_and_job0(jobs, L);
    int job = -1;
    for (int it = blockIdx.x; it < l.n; it += gridDim.x) {
        const WorkItem wi = l.items ? l.items[it] : WorkItem{0, it};
        const JobDev &J = jobs[wi.job];
        JobState *const st = J.st;
        const int W = J.W, rpc = J.rpc, y0 = wi.tile * rpc, nr = min(rpc, J.H - y0), n = nr * W;
        const size_t base = (size_t)y0 * W;
        const float2 *const X = J.X + base, *const gtw = J.prow.tw;
        const uint8_t *const mask = J.mask + base;
        const bool other = job != wi.job;
        const int word = other ? mx_plan_word(J.prow) : 0;
        if (job < 0) pdl_wait();
        const int oa = 0, ob = mx_row_pad(rpc * W), ot = 2 * ob + rpc * W;
        float2 xv[V];
#pragma unroll
        for (int m = 0; m < V; ++m) {
            const int i = threadIdx.x + m * T;
            if (i < n) xv[m] = X[i];
        }
        if (other)
            for (int i = threadIdx.x; i < W; i += T) cp_async8(sm + ot + i, gtw + i);
        uint8_t mk[V];
#pragma unroll
        for (int m = 0; m < V; ++m) {
            const int i = threadIdx.x + m * T;
            mk[m] = i < n ? mask[i] : 0;
        }
        // (a job that ended by its count has gone one cycle past the tables)
        const int stop = st->stop, c = min(st->cycle, J.n_cycles);
        const int K = J.ntaps[c];
        if (threadIdx.x < kTapStride) wsm[threadIdx.x] = J.weights[(size_t)c * kTapStride + threadIdx.x];
        if (other) mx_store_plan(&sp, word);
        job = wi.job;
#pragma unroll
        for (int m = 0; m < V; ++m) {
            const int i = threadIdx.x + m * T;
            if (i < n) sm[oa + mx_row_at(i)] = make_float2(xv[m].x, -xv[m].y);
        }
        cp_async_wait();
        __syncthreads();
        if (stop) continue;
        if (wi.tile == 0 && threadIdx.x == 0) st->max_bits = 0u;
        const int r = mx_fft<0, T>(oa, ob, ot, sp, nr, true);
        if (it + (int)gridDim.x >= l.n) pdl_trigger();
        float *const nrm = reinterpret_cast<float *>(sm + oa + ob - r);
        double tot = 0.0, cnt = 0.0;
#pragma unroll
        for (int m = 0; m < V; ++m) {
            const int i = threadIdx.x + m * T;
            if (i >= n) continue;
            float2 g = sm[r + mx_row_at(i)];
            g.y = -g.y;
            J.out[base + i] = g.x;
            if (dbg_gprime) dbg_gprime[base + i] = g;
            const float v = cnorm_ref(g);
            nrm[norm_at(i)] = v;
            if (c > 0 && mk[m]) {
                tot += (double)v;
                cnt += 1.0;
            }
        }
        block_sum2<T>(tot, cnt, red);   // includes barriers: nrm complete after it
        if (threadIdx.x == 0) {
            J.err_part[2 * wi.tile] = tot;
            J.err_part[2 * wi.tile + 1] = cnt;
        }
        // chunks of 8 neighbouring outputs; they leave through the transform's
        // buffer, coalesced whatever the width
        float *const out = reinterpret_cast<float *>(sm + r);
        const int cpr = (W + kRowChunk - 1) / kRowChunk;
        for (int q = threadIdx.x; q < nr * cpr; q += T) {
            const int row = q / cpr, x0 = (q - row * cpr) * kRowChunk;
            float sum[kRowChunk];
            row_chunk(sum, nrm, row * W, x0, W, wsm, K);
#pragma unroll
            for (int o = 0; o < kRowChunk; ++o)
                if (x0 + o < W) out[norm_at(row * W + x0 + o)] = sum[o];
        }
        __syncthreads();
#pragma unroll
        for (int m = 0; m < V; ++m) {
            const int i = threadIdx.x + m * T;
            if (i < n) J.hb[base + i] = out[norm_at(i)];
        }
        __syncthreads();
    }
}

template <int S>
__global__ void __launch_bounds__(kMxRowThreads, 3) k_fft_rows_mx(float2 *data, const __grid_constant__ FftPlanDev p,
                                                                  int H, int rpc)
{
    extern __shared__ float4 smem4[];
    float2 *const sm = reinterpret_cast<float2 *>(smem4);
    constexpr int T = kMxRowThreads, V = kMxRowElems / T;
    const int W = p.n, oa = 0, ob = mx_row_pad(rpc * W), ot = 2 * ob + rpc * W;
    const int y0 = blockIdx.x * rpc, nr = min(rpc, H - y0), n = nr * W;
    float2 *const X = data + (size_t)y0 * W;
    for (int i = threadIdx.x; i < W; i += T) cp_async8(sm + ot + i, p.tw + i);
    pdl_wait();
    float2 xv[V];
#pragma unroll
    for (int m = 0; m < V; ++m) {
        const int i = threadIdx.x + m * T;
        if (i < n) xv[m] = X[i];
    }
#pragma unroll
    for (int m = 0; m < V; ++m) {
        const int i = threadIdx.x + m * T;
        if (i < n) sm[oa + mx_row_at(i)] = make_float2(xv[m].x, S > 0 ? -xv[m].y : xv[m].y);
    }
    cp_async_wait();
    __syncthreads();
    const int r = mx_fft<0, T>(oa, ob, ot, p, nr, S > 0);
    pdl_trigger();
#pragma unroll
    for (int m = 0; m < V; ++m) {
        const int i = threadIdx.x + m * T;
        if (i >= n) continue;
        const float2 z = sm[r + mx_row_at(i)];
        X[i] = make_float2(z.x, S > 0 ? -z.y : z.y);
    }
}

// ---- columns ------------------------------------------------------------------
// mode 0 column pass (forward, modulus projection, inverse; see b_col),
// 1 column init (inverse of (M, 0)), 2 plain forward, 3 plain inverse
// request the tile (and the modulus of mode 0)
template <int MODE, int T, int C>
__device__ __forceinline__ void mx_col_request(const float2 *X, const float *M, int W, int H, int x0)
{
    extern __shared__ float4 smem4[];
    float2 *const sm = reinterpret_cast<float2 *>(smem4);
    constexpr int RS = T / C;   // rows per round of the block
    float *const smod = reinterpret_cast<float *>(sm + 2 * mx_col_pad<C>(H) + H);
    const int c = threadIdx.x % C, y_ = threadIdx.x / C;
    if (x0 + c < W) {
        const size_t col = x0 + c;
#pragma unroll 4
        for (int y = y_; y < H; y += RS) {
            if (MODE == 1) sm[mx_col_at<C>(y, c)] = make_float2(M[(size_t)y * W + col], 0.f);
            else if (MODE == 3) sm[mx_col_at<C>(y, c)] = make_float2(X[(size_t)y * W + col].x, -X[(size_t)y * W + col].y);
            else cp_async8(sm + mx_col_at<C>(y, c), X + (size_t)y * W + col);
            if (MODE == 0) cp_async4(smod + y * C + c, M + (size_t)y * W + col);
        }
    } else {
        for (int y = y_; y < H; y += RS) sm[mx_col_at<C>(y, c)] = make_float2(0.f, 0.f);
    }
}
// the tile's work once it has arrived
template <int MODE, int T, int C>
__device__ __forceinline__ void mx_col_run(float2 *X, int W, int H, int x0, const FftPlanDev &p, bool guard,
                                           bool last)
{
    extern __shared__ float4 smem4[];
    float2 *const sm = reinterpret_cast<float2 *>(smem4);
    constexpr int RS = T / C;
    const int ob = mx_col_pad<C>(H), ot = 2 * ob;
    const float *const smod = reinterpret_cast<const float *>(sm + ot + H);
    const int c = threadIdx.x % C, y_ = threadIdx.x / C;
    const bool ok = x0 + c < W;
    int r = 0;
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
        if (last && h == 1) pdl_trigger();
        r = mx_fft<C, T>(r, ob - r, ot, p, C, MODE == 1 || MODE == 3 || h == 1);
        if (MODE != 0 || h == 1) break;
        if (ok) {
#pragma unroll 4
            for (int y = y_; y < H; y += RS) {
                const float2 g = sm[r + mx_col_at<C>(y, c)];
                const float f = modulus_factor(smod[y * C + c], g, guard);
                sm[r + mx_col_at<C>(y, c)] = make_float2(__fmul_rn(g.x, f), -__fmul_rn(g.y, f));
            }
        }
        __syncthreads();
    }
    if (ok) {
#pragma unroll 4
        for (int y = y_; y < H; y += RS) {
            const float2 z = sm[r + mx_col_at<C>(y, c)];
            X[(size_t)y * W + x0 + c] = make_float2(z.x, MODE == 2 ? z.y : -z.y);
        }
    }
}

template <int MODE, int T, int C>
__global__ void __launch_bounds__(T, mx_col_blocks(T, C)) k_col_mx(const JobDev *jobs, const WorkList *L)
{
    extern __shared__ float4 smem4[];
    float2 *const sm = reinterpret_cast<float2 *>(smem4);
    __shared__ FftPlanDev sp;
    const WorkList l = list_and_job0(jobs, L);
    if (MODE == 0 && (int)blockIdx.x >= l.n) {
        hio_check_block<T>(jobs, l);
        return;
    }
    int job = -1;
    for (int it = blockIdx.x; it < l.n; it += gridDim.x) {
        const WorkItem wi = l.items ? l.items[it] : WorkItem{0, it};
        const JobDev &J = jobs[wi.job];
        const JobState *const st = J.st;
        const int W = J.W, H = J.H, x0 = wi.tile * C;
        float2 *const X = J.X;
        const float *const M = J.M;
        const float2 *const gtw = J.pcol.tw;
        const bool guard = J.mode == kModeShrinkWrap;
        const bool other = job != wi.job;
        const int word = other ? mx_plan_word(J.pcol) : 0;
        if (job < 0) pdl_wait();
        mx_col_request<MODE, T, C>(X, M, W, H, x0);
        if (other)
            for (int i = threadIdx.x; i < H; i += T) cp_async8(sm + 2 * mx_col_pad<C>(H) + i, gtw + i);
        const int stop = MODE == 0 ? st->stop : 0;   // (the check block may be setting it: decided as one)
        if (other) mx_store_plan(&sp, word);
        job = wi.job;
        cp_async_wait();
        if (__syncthreads_or(stop)) continue;
        mx_col_run<MODE, T, C>(X, W, H, x0, sp, guard, it + (int)gridDim.x >= l.n);
        __syncthreads();
    }
}

template <int S, int T, int C>
__global__ void __launch_bounds__(T, mx_col_blocks(T, C)) k_fft_cols_mx(float2 *data, const __grid_constant__ FftPlanDev p,
                                                                    int W, int)
{
    extern __shared__ float4 smem4[];
    float2 *const sm = reinterpret_cast<float2 *>(smem4);
    constexpr int MODE = S < 0 ? 2 : 3;
    const int H = p.n, x0 = blockIdx.x * C;
    pdl_wait();
    mx_col_request<MODE, T, C>(data, nullptr, W, H, x0);
    for (int i = threadIdx.x; i < H; i += T) cp_async8(sm + 2 * mx_col_pad<C>(H) + i, p.tw + i);
    cp_async_wait();
    __syncthreads();
    mx_col_run<MODE, T, C>(data, W, H, x0, p, true, false);
}

}  // namespace imr
