// rf_kern_post.cu -- FP64 post-processing of tallies on the device and the
// FP32 issue-rate probe.
//
// The reference divides the summed int tallies by the rays shot on the host in
// single precision (RayFactorCL/main.cpp:216-249).  Here the 64-bit tallies are
// normalised in FP64 on the GPU, and the same pass computes each row's largest
// binomial standard error sqrt(F(1-F)/rays) for the convergence loop.
#include <algorithm>
#include <cstdint>
#include <cuda_runtime.h>

#include "rf_internal.h"

namespace rf {

// F[i] = hits[i] / rays[row(i)]; NaN for rows without rays (0/0 in main.cpp:245).
__global__ void normalise_single_kernel(const unsigned long long *hits, const int64_t *rays, int n,
                                        double *F)
{
    const int64_t total = (int64_t)n * n;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = rays[i / n];
        F[i] = (double)hits[i] / (double)r;
    }
}

// The results of a single-scene trace straight into pinned host memory: tallies and F
// where wanted, the device's error flag and the mixed kernels' counters.  In place of
// four copies and a launch, each of which cost a small trace 5 to 10 us.
__global__ void finish_kernel(const unsigned long long *hits, const int64_t *rays, int n, unsigned long long *hits_out,
                              double *F_out, const int32_t *err, const unsigned long long *refined,
                              const unsigned long long *work, FinishHead *head)
{
    const int64_t total = (int64_t)n * n;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const unsigned long long h = hits[i];
        if (hits_out) hits_out[i] = h;
        if (F_out) F_out[i] = (double)h / (double)rays[i / n];
    }
    if (blockIdx.x == 0 && threadIdx.x < 8) {
        if (threadIdx.x == 0) {
            head->err = *err;
            head->refined = refined ? *refined : 0ull;
        }
        head->work[threadIdx.x] = work ? work[threadIdx.x] : 0ull;
    }
}

cudaError_t launch_finish(const unsigned long long *hits, const int64_t *rays, int n, unsigned long long *hits_out,
                          double *F_out, const int32_t *err, const unsigned long long *refined,
                          const unsigned long long *work, FinishHead *head, cudaStream_t st)
{
    const int64_t total = hits_out || F_out ? (int64_t)n * n : 1;
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(1024, (total + 255) / 256));
    finish_kernel<<<grid, 256, 0, st>>>(hits, rays, n, hits_out, F_out, err, refined, work, head);
    return cudaGetLastError();
}

cudaError_t launch_normalise_single(const unsigned long long *hits, const int64_t *rays, int n,
                                    double *F, cudaStream_t st)
{
    const int64_t total = (int64_t)n * n;
    int grid = (int)((total + 255) / 256);
    if (grid > 4096) grid = 4096;
    if (grid < 1) grid = 1;
    normalise_single_kernel<<<grid, 256, 0, st>>>(hits, rays, n, F);
    return cudaGetLastError();
}

// One warp per row of the batched tally: F, row standard error and the next
// round's budget.  A row converges when max_j sqrt(F(1-F)/rays) <= tol.  An
// unconverged row is given the rays its current estimate says it still needs,
// ceil(max_j F(1-F) / tol^2) - rays (rounded up to whole draws of 4 rays), at
// most round_rays per round; an underestimate is corrected by the next round.
__global__ void converge_step_kernel(const unsigned long long *hits, int64_t *rays,
                                     const int64_t *row_off, const int32_t *row_n, int64_t nrows,
                                     double *F, double tol, int64_t *next_rays, int64_t round_rays,
                                     int32_t *not_converged)
{
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= nrows) return;
    const int64_t off = row_off[warp];
    const int len = row_n[warp];
    const int64_t r = rays[warp];
    double worst = 0.0;  // max_j F(1-F)
    for (int j = lane; j < len; j += 32) {
        const double f = r > 0 ? (double)hits[off + j] / (double)r : 0.0;
        if (F) F[off + j] = r > 0 ? f : __longlong_as_double(0x7ff8000000000000ll);
        worst = fmax(worst, r > 0 ? f * (1.0 - f) : 1.0);
    }
    for (int o = 16; o; o >>= 1) worst = fmax(worst, __shfl_xor_sync(0xffffffffu, worst, o));
    if (lane == 0) {
        const bool more = r <= 0 || sqrt(worst / (double)r) > tol;
        int64_t add = 0;
        if (more) {
            const double need = r > 0 ? ceil(worst / (tol * tol)) - (double)r : (double)round_rays;
            add = need >= (double)round_rays ? round_rays : (int64_t)need;
            add = (add + 3) & ~(int64_t)3;
            if (add < 4) add = 4;
            if (add > round_rays) add = round_rays;
        }
        next_rays[warp] = add;
        if (more) atomicAdd(not_converged, 1);
    }
}

cudaError_t launch_converge_step(const unsigned long long *hits, int64_t *rays,
                                 const int64_t *row_off, const int32_t *row_n, int64_t nrows,
                                 double *F, double tol, int64_t *next_rays, int64_t round_rays,
                                 int32_t *not_converged, cudaStream_t st)
{
    const int64_t threads = nrows * 32;
    int grid = (int)((threads + 255) / 256);
    if (grid < 1) grid = 1;
    converge_step_kernel<<<grid, 256, 0, st>>>(hits, rays, row_off, row_n, nrows, F, tol, next_rays,
                                               round_rays, not_converged);
    return cudaGetLastError();
}

// One round of the convergence loop, planned on the device: every row with
// next[r] > 0 rays to add becomes a segment continuing its stream at
// rays_total[r]; chunks, sized for the round's rays (the last rounds' few rows would
// otherwise be a few long chunks on as many SMs), are numbered across segments; the
// work queue is reset.
__global__ void plan_round_kernel(int64_t nrows, const int32_t *row_scene, const int32_t *row_emitter,
                                  int64_t *rays_total, const int64_t *next, Segment *seg, int32_t *d_nseg,
                                  int64_t *d_total, unsigned long long *queue, int sms, int32_t *d_chunk)
{
    __shared__ int64_t s_chunks[1024];
    __shared__ int32_t s_nz[1024];
    const int tid = threadIdx.x, T = blockDim.x;
    const int64_t lo = nrows * tid / T, hi = nrows * (tid + 1) / T;
    int64_t draws = 0;
    for (int64_t r = lo; r < hi; ++r)
        if (next[r] > 0) draws += (next[r] + 3) >> 2;
    s_chunks[tid] = draws;
    __syncthreads();
    for (int o = T / 2; o; o >>= 1) {
        if (tid < o) s_chunks[tid] += s_chunks[tid + o];
        __syncthreads();
    }
    const int chunk_draws = chunk_for(s_chunks[0], sms, 1024);
    __syncthreads();
    int64_t chunks = 0;
    int32_t nz = 0;
    for (int64_t r = lo; r < hi; ++r) {
        const int64_t add = next[r];
        if (add <= 0) continue;
        const int64_t b = rays_total[r], g0 = b >> 2, g1 = (b + add + 3) >> 2;
        chunks += (g1 - g0 + chunk_draws - 1) / chunk_draws;
        ++nz;
    }
    s_chunks[tid] = chunks;
    s_nz[tid] = nz;
    __syncthreads();
    for (int o = 1; o < T; o <<= 1) {  // inclusive Hillis-Steele scan
        const int64_t c = tid >= o ? s_chunks[tid - o] : 0;
        const int32_t z = tid >= o ? s_nz[tid - o] : 0;
        __syncthreads();
        s_chunks[tid] += c;
        s_nz[tid] += z;
        __syncthreads();
    }
    int64_t cpos = s_chunks[tid] - chunks;
    int32_t spos = s_nz[tid] - nz;
    for (int64_t r = lo; r < hi; ++r) {
        const int64_t add = next[r];
        if (add <= 0) continue;
        const int64_t b = rays_total[r], g0 = b >> 2, g1 = (b + add + 3) >> 2;
        Segment sg;
        sg.emitter = row_emitter[r];
        sg.scene = row_scene[r];
        sg.ray_begin = b;
        sg.ray_end = b + add;
        sg.chunk_begin = cpos;
        seg[spos++] = sg;
        cpos += (g1 - g0 + chunk_draws - 1) / chunk_draws;
        rays_total[r] = b + add;
    }
    if (tid == T - 1) {
        *d_nseg = s_nz[T - 1];
        *d_total = s_chunks[T - 1];
        *queue = 0ull;
        *d_chunk = chunk_draws;
    }
}

cudaError_t launch_plan_round(int64_t nrows, const int32_t *row_scene, const int32_t *row_emitter,
                              int64_t *rays_total, const int64_t *next, Segment *seg, int32_t *d_nseg,
                              int64_t *d_total, unsigned long long *queue, int sms, int32_t *d_chunk, cudaStream_t st)
{
    plan_round_kernel<<<1, 1024, 0, st>>>(nrows, row_scene, row_emitter, rays_total, next, seg, d_nseg,
                                          d_total, queue, sms, d_chunk);
    return cudaGetLastError();
}

// Loop control of the convergence graph: one more round while some row is
// above the tolerance and fewer than max_rounds rounds ran.
__global__ void decide_round_kernel(int32_t *flags, int32_t max_rounds, cudaGraphConditionalHandle h)
{
    const int32_t rounds = flags[1] + 1;
    flags[1] = rounds;
    const bool more = flags[0] > 0 && rounds < max_rounds;
    flags[0] = 0;
    cudaGraphSetConditional(h, more ? 1u : 0u);
}

cudaError_t launch_decide_round(int32_t *flags, int32_t max_rounds, unsigned long long handle,
                                cudaStream_t st)
{
    decide_round_kernel<<<1, 1, 0, st>>>(flags, max_rounds, (cudaGraphConditionalHandle)handle);
    return cudaGetLastError();
}

__device__ __forceinline__ void atomic_max_double(double *a, double v)
{
    // non-negative doubles order like their bit patterns
    atomicMax(reinterpret_cast<unsigned long long *>(a), (unsigned long long)__double_as_longlong(v));
}

// out2[0] = max_i |sum_j F_ij - 1|; out2[1] = max over pairs with both entries
// non-zero of |A_i F_ij - A_j F_ji| / max(A_i F_ij, A_j F_ji).  Bound by FP64
// operations (two a clock on an SM): each pair is looked at once, its ratio compared
// by cross products and divided only at the end.  A block takes four rows, so that
// the transposed entries it reads fill their 32-byte sectors.
constexpr int kCheckRows = 4;
__global__ void __launch_bounds__(256) check_F_kernel(const double *F, const double *areas, int n, double *out2)
{
    const int r = threadIdx.x % kCheckRows, q = threadIdx.x / kCheckRows, i = blockIdx.x * kCheckRows + r;
    double s = 0.0, num = 0.0, den = 1.0;
    if (i < n) {
        const double ai = areas ? areas[i] : 0.0;
        for (int j = q; j < n; j += 256 / kCheckRows) {
            const double fij = F[(int64_t)i * n + j];
            s += fij;
            if (areas && j > i && fij > 0.0) {
                const double fji = F[(int64_t)j * n + i];
                if (fji > 0.0) {
                    const double a = ai * fij, b = areas[j] * fji, d = fabs(a - b), m = fmax(a, b);
                    if (d * den > num * m) {
                        num = d;
                        den = m;
                    }
                }
            }
        }
    }
    __shared__ double ss[256], sw[256];
    ss[threadIdx.x] = s;
    sw[threadIdx.x] = num / den;
    __syncthreads();
    for (int o = 128; o >= kCheckRows; o >>= 1) {
        if (threadIdx.x < o) {
            ss[threadIdx.x] += ss[threadIdx.x + o];
            sw[threadIdx.x] = fmax(sw[threadIdx.x], sw[threadIdx.x + o]);
        }
        __syncthreads();
    }
    if (threadIdx.x < kCheckRows && i < n) {
        atomic_max_double(&out2[0], fabs(ss[threadIdx.x] - 1.0));
        atomic_max_double(&out2[1], sw[threadIdx.x]);
    }
}

cudaError_t launch_check_F(const double *F, const double *areas, int n, double *out2, cudaStream_t st)
{
    cudaError_t e = cudaMemsetAsync(out2, 0, 2 * sizeof(double), st);
    if (e != cudaSuccess) return e;
    check_F_kernel<<<(n + kCheckRows - 1) / kCheckRows, 256, 0, st>>>(F, areas, n, out2);
    return cudaGetLastError();
}

// Reciprocity and summation enforcement (FP64).  G_ij = (A_i F_ij + A_j F_ji)/2
// is the symmetric exchange matrix closest to the tallies (reciprocity holds
// exactly for any symmetric G).  For a closed enclosure the rows must also sum
// to 1: a symmetric scaling X G X with X = diag(x) keeps the symmetry, and x is
// found by the symmetric Sinkhorn iteration x_i <- sqrt(x_i A_i / (G x)_i).
//
// One cooperative launch: block b owns a run of consecutive rows, keeps them in
// shared memory when they fit (RES; n up to about 2000), forms G, iterates and writes
// the scaled rows.  A round is n^2 FP64 multiply-adds (two a clock on an SM: 0.3 us
// at n = 412 over the chip) and an exchange of x through L2, without a barrier: an
// element is published with its round as one 16-byte word, and its readers wait for
// the round they need.  Two buffers suffice: who publishes round r + 2 has read all of
// round r + 1, so everyone has read round r.  A row's sum keeps the order of a
// 256-thread block's tree (partial sums t, t + 256, ...; halves added), a warp holding
// eight partials per lane; one warp then takes the roots of all rows of the block.
// n = 412, 56 rounds: 0.22 ms (7400 clocks a round: 2600 row sums, 1700 root and
// quotient, 3100 exchange), 0.34 for the call; as a launch and a memset per round with a
// host check every eight, 0.38 ms of kernels and 0.85 for the call.
struct SmoothState {
    double final_err;
    int iters;
    int gave_up;  // some wait ran out of time
};
struct __align__(16) Tagged {
    double v;
    unsigned long long round;
};

__device__ __forceinline__ void publish(Tagged *p, double v, unsigned long long round)
{
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
                 "l"(__double_as_longlong(v)), "l"(round)
                 : "memory");
}

// The value published for `round` at p; false after about two seconds (2^32 clocks)
// without it, or when another wait gave up.
__device__ __forceinline__ bool await(const Tagged *p, unsigned long long round, SmoothState *st, double &v)
{
    long long bits, t0 = 0;
    unsigned long long have;
    for (int spin = 0;; ++spin) {
        asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
                     : "=l"(bits), "=l"(have)
                     : "l"(p)
                     : "memory");
        if (have == round) break;
        if (spin == 0) t0 = clock64();
        if ((spin & 63) == 63 &&
            (*reinterpret_cast<volatile int *>(&st->gave_up) || clock64() - t0 > (1ll << 32))) {
            *reinterpret_cast<volatile int *>(&st->gave_up) = 1;
            return false;
        }
    }
    v = __longlong_as_double(bits);
    return true;
}

constexpr int kSmoothThreads = 512;
constexpr int kSmoothRows = 256;  // row sums of a pass: rows of a block are taken in runs of this many

template <bool RES>
__global__ void __launch_bounds__(kSmoothThreads, 1)
    smooth_kernel(const double *F, const double *A, int n, int closed, int max_iter, double tol, double *G, double *xg,
                  Tagged *xbuf, Tagged *ebuf, double *F_out, SmoothState *st)
{
    extern __shared__ double s_rows[];  // RES: this block's rows of G, then x
    __shared__ double s_sum[kSmoothRows];
    __shared__ double s_err[kSmoothThreads / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = kSmoothThreads / 32;
    const int i0 = (int)((int64_t)n * blockIdx.x / gridDim.x), i1 = (int)((int64_t)n * (blockIdx.x + 1) / gridDim.x);
    const int rows = i1 - i0;
    double *g = RES ? s_rows : G + (int64_t)i0 * n;
    double *x = RES ? s_rows + (int64_t)rows * n : xg + (int64_t)blockIdx.x * n;  // this block's copy of x
    // rows fastest: the transposed entries of a block are contiguous
    for (int64_t k = tid; k < (int64_t)rows * n; k += kSmoothThreads) {
        const int j = (int)(k / rows), i = i0 + (int)(k % rows);
        const double a = F[(int64_t)i * n + j], b = F[(int64_t)j * n + i];
        const double fa = (a == a) ? a : 0.0, fb = (b == b) ? b : 0.0;  // rows without rays: 0
        g[(int64_t)(i - i0) * n + j] = 0.5 * (A[i] * fa + A[j] * fb);
    }
    if (closed) {
        for (int j = tid; j < n; j += kSmoothThreads) x[j] = 1.0;
        __syncthreads();
        for (int it = 0; it < max_iter; ++it) {
            const bool check = (it & 7) == 7 || it + 1 == max_iter;
            const unsigned long long round = it + 1;
            Tagged *xb = xbuf + (int64_t)(it & 1) * n, *eb = ebuf + (int64_t)((it >> 3) & 1) * n;
            for (int r0 = 0; r0 < rows; r0 += kSmoothRows) {
                const int cnt = min(kSmoothRows, rows - r0);
                for (int r = warp; r < cnt; r += nwarps) {
                    const double *gr = g + (int64_t)(r0 + r) * n;
                    double p[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
                    for (int b = lane; b < n; b += 256)  // eight independent loads and chains
#pragma unroll
                        for (int k = 0; k < 8; ++k)
                            if (b + 32 * k < n) p[k] += gr[b + 32 * k] * x[b + 32 * k];
#pragma unroll
                    for (int h = 4; h; h >>= 1)
#pragma unroll
                        for (int k = 0; k < h; ++k) p[k] += p[k + h];
                    double s = p[0];
#pragma unroll
                    for (int o = 16; o; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
                    if (lane == 0) s_sum[r] = s;
                }
                __syncthreads();
                for (int r = tid; r < cnt; r += kSmoothThreads) {
                    const int i = i0 + r0 + r;
                    const double s = s_sum[r], xi = x[i], a = A[i];
                    double xn = xi, e = 0.0;  // a surface that sees nothing keeps its row
                    if (s > 0.0 && a > 0.0) {
                        xn = sqrt(xi * a / s);
                        if (check) e = fabs(xi * s / a - 1.0);
                    }
                    publish(xb + i, xn, round);
                    if (check) publish(eb + i, e, round);
                }
                if (r0 + kSmoothRows < rows) __syncthreads();
            }
            __syncthreads();  // every row's sum is formed: x may change
            bool ok = true;
            double worst = 0.0;
            for (int j = tid; j < n && ok; j += kSmoothThreads) {
                double v = 0.0;
                ok = await(xb + j, round, st, v);
                x[j] = v;
                if (check && ok) {
                    ok = await(eb + j, round, st, v);
                    worst = fmax(worst, v);
                }
            }
            if (check) {
#pragma unroll
                for (int o = 16; o; o >>= 1) worst = fmax(worst, __shfl_xor_sync(0xffffffffu, worst, o));
                if (lane == 0) s_err[warp] = worst;
            }
            if (__syncthreads_or(!ok)) return;
            if (check) {
                double e = 0.0;
#pragma unroll
                for (int k = 0; k < nwarps; ++k) e = fmax(e, s_err[k]);
                if (blockIdx.x == 0 && tid == 0) {
                    st->iters = it + 1;
                    st->final_err = e;
                }
                if (e <= tol) break;  // the same in every block
            }
        }
    }
    __syncthreads();
    for (int64_t k = tid; k < (int64_t)rows * n; k += kSmoothThreads) {
        const int r = (int)(k / n), j = (int)(k % n), i = i0 + r;
        const double v = g[k];
        F_out[(int64_t)i * n + j] = A[i] > 0.0 ? (closed ? x[i] * v * x[j] : v) / A[i] : 0.0;
    }
}

// Workspace in bytes: two 16-byte-tagged buffers of x and of the errors, the state,
// and, where a block's rows do not fit shared memory, G and the blocks' copies of x.
constexpr size_t kSmoothShared = 216 * 1024;  // most that a block's rows and x take
static bool smooth_resident(int n, int grid)
{
    const size_t rows = (n + grid - 1) / grid;
    return (rows + 1) * n * sizeof(double) <= kSmoothShared;
}
size_t smooth_bytes(int n, int sms)
{
    const int grid = std::min(n, sms);
    const size_t tagged = 4 * (size_t)n * sizeof(Tagged) + 64;
    return tagged + (smooth_resident(n, grid) ? 0 : ((size_t)n + grid) * n * sizeof(double));
}

cudaError_t launch_smooth(const double *F, const double *A, int n, int closed, int max_iter, double tol, void *work,
                          double *F_out, int sms, int *iters, double *final_err, bool *gave_up, cudaStream_t st)
{
    const int grid = std::min(n, sms);
    const bool resident = smooth_resident(n, grid);
    Tagged *xbuf = static_cast<Tagged *>(work), *ebuf = xbuf + 2 * (size_t)n;
    SmoothState *ds = reinterpret_cast<SmoothState *>(ebuf + 2 * (size_t)n);
    double *G = reinterpret_cast<double *>(ds) + 8, *xg = G + (size_t)n * n;
    cudaError_t e = cudaMemsetAsync(work, 0, 4 * (size_t)n * sizeof(Tagged) + 64, st);  // no round published
    if (e != cudaSuccess) return e;
    const size_t rows = (n + grid - 1) / grid, smem = resident ? (rows + 1) * n * sizeof(double) : 0;
    const void *k = resident ? (const void *)smooth_kernel<true> : (const void *)smooth_kernel<false>;
    // (the largest launch's size, whatever this one takes: the attribute is the function's, and
    // another thread's context may launch it at the same time)
    if ((e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, resident ? (int)kSmoothShared : 0)) != cudaSuccess)
        return e;
    void *args[] = {&F, &A, &n, &closed, &max_iter, &tol, &G, &xg, &xbuf, &ebuf, &F_out, &ds};
    if ((e = cudaLaunchCooperativeKernel(k, dim3(grid), dim3(kSmoothThreads), args, smem, st)) != cudaSuccess) return e;
    SmoothState h{};
    if ((e = cudaMemcpyAsync(&h, ds, sizeof h, cudaMemcpyDeviceToHost, st)) != cudaSuccess) return e;
    if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return e;
    *iters = h.iters;
    *final_err = h.final_err;
    *gave_up = h.gave_up != 0;
    return cudaSuccess;
}

// Eight independent FMA chains per thread: the FP32 issue roofline.
__global__ void fp32_probe_kernel(float *out, int iters)
{
    float a0 = threadIdx.x * 1e-7f, a1 = a0 + 1e-7f, a2 = a0 + 2e-7f, a3 = a0 + 3e-7f;
    float a4 = a0 + 4e-7f, a5 = a0 + 5e-7f, a6 = a0 + 6e-7f, a7 = a0 + 7e-7f;
    const float m = 0.999999f, c = 1e-7f;
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int u = 0; u < 16; ++u) {
            a0 = __fmaf_rn(a0, m, c); a1 = __fmaf_rn(a1, m, c);
            a2 = __fmaf_rn(a2, m, c); a3 = __fmaf_rn(a3, m, c);
            a4 = __fmaf_rn(a4, m, c); a5 = __fmaf_rn(a5, m, c);
            a6 = __fmaf_rn(a6, m, c); a7 = __fmaf_rn(a7, m, c);
        }
    }
    const float s = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
    if (s == 12345.678f) out[blockIdx.x * blockDim.x + threadIdx.x] = s;  // keeps the chains live
}

cudaError_t launch_fp32_probe(float *out, int iters, int grid, int block, cudaStream_t st)
{
    fp32_probe_kernel<<<grid, block, 0, st>>>(out, iters);
    return cudaGetLastError();
}

}  // namespace rf
