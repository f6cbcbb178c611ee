// solver.cu -- red-black SOR for the reference's Poisson problem on sm_103a.
//
// Reference: poisson_solver / patial_relax, src/solver.cpp:12-148.  The
// reference relaxes lexicographically (Gauss-Seidel order) with
// omega = 2/(1+pi/width) and stops when one sweep's max |delta| drops below a
// threshold.  Here every sweep is two half sweeps over the red ((x+y) even)
// and black cells, which have no neighbours of their own colour, so each half
// sweep is one fully parallel kernel.  Red-black SOR with the same omega has
// the same asymptotic rate as the lexicographic ordering (both are consistent
// orderings); intermediate iterates differ, the fixed point is the same.
//
// Two stop tests: the reference's max |delta| (checked after every sweep by
// the last block of the black half sweep) and a relative FP64 residual
// ||b - L phi|| / ||b|| checked every `check_every` sweeps.
//
// Two precisions: FP64 sweeps on phi, or FP32 sweeps on the error equation
// L e = r with the residual r = b - L(phi + e) and the update phi += e done in
// FP64 every `refine_every` sweeps (defect correction).  SOR is a stationary
// iteration, so restarting it on the refreshed residual from e = 0 changes
// nothing in exact arithmetic; FP32 only limits how far e may be pushed
// between refreshes.
//
// Sweeps are issued as CUDA-graph chunks; the stop flags live in device memory
// and make the remaining kernels of a chunk return at once, so the host reads
// the control block once per chunk and launches the next chunk speculatively.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "solver.cuh"
#include "sor_persist.cuh"
#include "sor_cluster.cuh"
#include "sor_blocks.cuh"
#include "sor_blocks64.cuh"
#include "sor_passes.cuh"
#include "sor_resident.cuh"
#include "refresh.cuh"
#include "sor_quads.cuh"

namespace pcd {

namespace {

constexpr int kThreads = 256;
constexpr int kResidualBlocksMax = 1216;  // 152 SMs x 8

__device__ __forceinline__ int vol_load(const int *p) { return *(volatile const int *)p; }

// ---------------------------------------------------------------------------
// Neighbour-validity mask: bit0 left, bit1 up, bit2 right, bit3 down (inside
// the grid and b not NaN, solver.cpp:29-44); bit4 set when b itself is NaN.
// ---------------------------------------------------------------------------
__global__ void k_mask(const double *__restrict__ b, uint8_t *__restrict__ mask, int W, int H, int ld,
                       Ctl *ctl)
{
    long n = (long)W * H;
    int nan_local = 0;
    for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x) {
        int y = (int)(t / W), x = (int)(t - (long)y * W);
        long i = (long)y * ld + x;
        uint8_t m = 0;
        if (x > 0 && !isnan(b[i - 1])) m |= 1;
        if (y > 0 && !isnan(b[i - ld])) m |= 2;
        if (x < W - 1 && !isnan(b[i + 1])) m |= 4;
        if (y < H - 1 && !isnan(b[i + ld])) m |= 8;
        if (isnan(b[i])) { m |= 16; nan_local++; }
        mask[i] = m;
    }
    if (nan_local) atomicAdd(&ctl->nan_cells, nan_local);
}

template <typename T, bool MASKED>
__device__ __forceinline__ void gather(const T *__restrict__ phi, const uint8_t *__restrict__ mask, long i, int x,
                                       int y, int W, int H, int ld, T &sum, T &cnt)
{
    sum = T(0);
    cnt = T(0);
    if (MASKED) {
        const uint8_t m = mask[i];
        if (m & 1) { cnt += T(1); sum += phi[i - 1]; }
        if (m & 2) { cnt += T(1); sum += phi[i - ld]; }
        if (m & 4) { cnt += T(1); sum += phi[i + 1]; }
        if (m & 8) { cnt += T(1); sum += phi[i + ld]; }
    } else {
        if (x > 0) { cnt += T(1); sum += phi[i - 1]; }
        if (y > 0) { cnt += T(1); sum += phi[i - ld]; }
        if (x < W - 1) { cnt += T(1); sum += phi[i + 1]; }
        if (y < H - 1) { cnt += T(1); sum += phi[i + ld]; }
    }
}

// omega/cnt from the host-divided table, selected without dynamic indexing
// (which would place the argument struct in local memory).
template <typename T>
__device__ __forceinline__ T omega_over_cnt(const SolveArgs &a, int cnt)
{
    if (sizeof(T) == 8)
        return (T)(cnt == 4 ? a.w64[4] : cnt == 3 ? a.w64[3] : cnt == 2 ? a.w64[2] : cnt == 1 ? a.w64[1] : a.w64[0]);
    return (T)(cnt == 4 ? a.w32[4] : cnt == 3 ? a.w32[3] : cnt == 2 ? a.w32[2] : cnt == 1 ? a.w32[1] : a.w32[0]);
}

// One half sweep over the cells of `color`: delta = omega/cnt*(sum - cnt*v - b)
// (solver.cpp:47), phi += delta.  TRACK keeps the sweep's max |delta|.
template <typename T, bool MASKED, bool TRACK>
__global__ void __launch_bounds__(kThreads)
    k_rb_half(T *__restrict__ phi, const T *__restrict__ rhs, const uint8_t *__restrict__ mask, Ctl *ctl,
              SolveArgs a, int color, int last_half)
{
    if (vol_load(&ctl->halt)) return;
    const int half = (a.W + 1) >> 1;
    const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
    double m = 0.0;
    if (idx < (long)a.H * half) {
        const int y = (int)(idx / half);
        const int x = 2 * (int)(idx - (long)y * half) + ((y + color) & 1);
        if (x < a.W) {
            const long i = (long)y * a.ld + x;
            T sum, cnt;
            gather<T, MASKED>(phi, mask, i, x, y, a.W, a.H, a.ld, sum, cnt);
            const T v = phi[i];
            const T w = omega_over_cnt<T>(a, (int)cnt);
            const T delta = w * (sum - cnt * v - rhs[i]);
            phi[i] = v + delta;
            if (TRACK) {
                double ad = fabs((double)delta);
                m = ad > 0.0 ? ad : 0.0;  // NaN deltas never raise the max (solver.cpp:51)
            }
        }
    }
    if (!TRACK && !last_half) return;
    if (TRACK) {
        double v[1] = {m};
        block_reduce<1, 1u>(v);
        m = v[0];
    }
    if (threadIdx.x == 0) {
        if (TRACK && m > 0.0) atomicMax(&ctl->maxbits, (unsigned long long)__double_as_longlong(m));
        if (last_half) {
            __threadfence();
            unsigned t = atomicAdd(&ctl->blocks_done, 1u);
            if (t == gridDim.x - 1) {
                __threadfence();
                end_of_sweep(ctl, a);
            }
        }
    }
}

// Last-block finalisation of a residual reduction: sums the per-block
// partials in a fixed order (deterministic), stores the norms and applies the
// relative-residual stop test when `test` is set.
__device__ void finalize_residual(Ctl *ctl, const double *partials, int nblk, const SolveArgs &a, int test,
                                  int with_b)
{
    double v[3] = {0.0, 0.0, 0.0};
    for (int k = threadIdx.x; k < nblk; k += blockDim.x) {
        v[0] += partials[3 * k];
        v[1] += partials[3 * k + 1];
        v[2] = fmax(v[2], partials[3 * k + 2]);
    }
    block_reduce<3, 4u>(v);
    if (threadIdx.x == 0) {
        volatile Ctl *c = ctl;
        double rn = sqrt(v[0]);
        if (with_b) c->bnorm = sqrt(v[1]);
        double bn = c->bnorm;
        c->rnorm = rn;
        c->rmax = v[2];
        double rel = bn > 0.0 ? rn / bn : rn;
        c->rel = rel;
        c->checks = c->checks + 1;
        if (test && a.stop == PCD_STOP_REL_RESIDUAL && rel <= a.tol) {
            c->converged = 1;
            c->halt = 1;
        }
        c->blocks_done_r = 0;
        __threadfence();
    }
}

__device__ __forceinline__ bool last_block(Ctl *ctl)
{
    __shared__ bool is_last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        unsigned t = atomicAdd(&ctl->blocks_done_r, 1u);
        is_last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (is_last) __threadfence();
    return is_last;
}

// FP64 residual r = b - L phi over non-NaN cells; partial sums of r^2, b^2
// and max |r|.  `test`: apply the stop test (loop checks); `skip_halted`:
// return at once when the solve already halted.
template <bool MASKED>
__global__ void __launch_bounds__(kThreads)
    k_residual64(const double *__restrict__ phi, const double *__restrict__ b, const uint8_t *__restrict__ mask,
                 Ctl *ctl, double *partials, SolveArgs a, int test, int with_b, int skip_halted,
                 double *__restrict__ rout = nullptr)
{
    if (skip_halted && vol_load(&ctl->halt)) return;
    const long n = (long)a.W * a.H;
    double v[3] = {0.0, 0.0, 0.0};
    for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x) {
        const int y = (int)(t / a.W), x = (int)(t - (long)y * a.W);
        const long i = (long)y * a.ld + x;
        const double bi = b[i];
        if (isnan(bi)) continue;
        double sum, cnt;
        gather<double, MASKED>(phi, mask, i, x, y, a.W, a.H, a.ld, sum, cnt);
        const double r = bi - (sum - cnt * phi[i]);
        if (rout) rout[i] = r;
        v[0] += r * r;
        v[1] += bi * bi;
        v[2] = nan_skip_max(v[2], fabs(r));
    }
    block_reduce<3, 4u>(v);
    if (threadIdx.x == 0) {
        partials[3 * blockIdx.x] = v[0];
        partials[3 * blockIdx.x + 1] = v[1];
        partials[3 * blockIdx.x + 2] = v[2];
    }
    if (last_block(ctl)) finalize_residual(ctl, partials, gridDim.x, a, test, with_b);
}

// Mixed precision: r = b - L(phi + e) in FP64 (e widened exactly), written to
// r32 as the next right-hand side of the FP32 correction sweeps.
template <bool MASKED>
__global__ void __launch_bounds__(kThreads)
    k_refine_residual(const double *__restrict__ phi, const float *__restrict__ e, const double *__restrict__ b,
                      const uint8_t *__restrict__ mask, float *__restrict__ r32, Ctl *ctl, double *partials,
                      SolveArgs a, int with_b)
{
    if (vol_load(&ctl->done)) return;
    const long n = (long)a.W * a.H;
    double v[3] = {0.0, 0.0, 0.0};
    for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x) {
        const int y = (int)(t / a.W), x = (int)(t - (long)y * a.W);
        const long i = (long)y * a.ld + x;
        const double bi = b[i];
        double sum = 0.0, cnt = 0.0;
        if (MASKED) {
            const uint8_t m = mask[i];
            if (m & 1) { cnt += 1.0; sum += phi[i - 1] + (double)e[i - 1]; }
            if (m & 2) { cnt += 1.0; sum += phi[i - a.ld] + (double)e[i - a.ld]; }
            if (m & 4) { cnt += 1.0; sum += phi[i + 1] + (double)e[i + 1]; }
            if (m & 8) { cnt += 1.0; sum += phi[i + a.ld] + (double)e[i + a.ld]; }
        } else {
            if (x > 0) { cnt += 1.0; sum += phi[i - 1] + (double)e[i - 1]; }
            if (y > 0) { cnt += 1.0; sum += phi[i - a.ld] + (double)e[i - a.ld]; }
            if (x < a.W - 1) { cnt += 1.0; sum += phi[i + 1] + (double)e[i + 1]; }
            if (y < a.H - 1) { cnt += 1.0; sum += phi[i + a.ld] + (double)e[i + a.ld]; }
        }
        const double xi = phi[i] + (double)e[i];
        const double r = bi - (sum - cnt * xi);
        r32[i] = (float)r;
        if (isnan(bi)) continue;
        v[0] += r * r;
        v[1] += bi * bi;
        v[2] = nan_skip_max(v[2], fabs(r));
    }
    block_reduce<3, 4u>(v);
    if (threadIdx.x == 0) {
        partials[3 * blockIdx.x] = v[0];
        partials[3 * blockIdx.x + 1] = v[1];
        partials[3 * blockIdx.x + 2] = v[2];
    }
    if (last_block(ctl)) finalize_residual(ctl, partials, gridDim.x, a, 1, with_b);
}

// Mixed precision: phi += e, e = 0.  The last block marks the solve done once
// the sweeps have halted (the correction that halted them is now in phi).
__global__ void __launch_bounds__(kThreads)
    k_refine_update(double *__restrict__ phi, float *__restrict__ e, Ctl *ctl, SolveArgs a)
{
    if (vol_load(&ctl->done)) return;
    const long n = (long)a.W * a.H;
    for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x) {
        const int y = (int)(t / a.W), x = (int)(t - (long)y * a.W);
        const long i = (long)y * a.ld + x;
        phi[i] += (double)e[i];
        e[i] = 0.0f;
    }
    if (last_block(ctl)) {
        if (threadIdx.x == 0) {
            volatile Ctl *c = ctl;
            if (c->halt) c->done = 1;
            c->blocks_done_r = 0;
            __threadfence();
        }
    }
}


// ---------------------------------------------------------------------------
// Fused red+black sweep for grids that live in HBM (no NaN cells).
//
// Block s walks down its stripe of rows [y0, y1): at step j it relaxes the red
// cells of row y0+j and then the black cells of row y0+j-1.  A red cell needs
// the black rows y-1, y, y+1 as they were before the sweep, and a black cell
// needs the new red rows y-1, y, y+1; walking down the stripe gives exactly
// that order, with one block barrier per step.  The black cells of the first
// and last row of every stripe depend on a neighbouring stripe's red row, so a
// second kernel relaxes those after all stripes finished.  The result is
// exactly one red-black SOR sweep, and phi and b cross HBM once per sweep
// (24 B per cell in FP64, 12 B in FP32) instead of twice.
constexpr int kStripeThreads = 512;

__device__ __forceinline__ void prefetch_l2(const void *p)
{
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// One colour of row y.  All loads of a thread's cells are issued before any
// store: a cell's neighbours have the other colour, so no cell of this row
// reads what another cell of it writes, and batching lets the DRAM latency of
// the cells overlap instead of serialising behind each store.
constexpr int kRowCellsMax = 8;  // cells per thread per row: W <= 2 * 8 * kStripeThreads

template <typename T, bool TRACK, int CELLS>
__device__ __forceinline__ double relax_row(T *__restrict__ phi, const T *__restrict__ rhs, const SolveArgs &a,
                                            int y, int color)
{
    const int W = a.W, H = a.H, ld = a.ld;
    const int off = (y + color) & 1;
    const long rowi = (long)y * ld;
    T sum[CELLS], v[CELLS], r[CELLS];
    int cnt[CELLS];
#pragma unroll
    for (int j = 0; j < CELLS; j++) {
        const int x = 2 * (threadIdx.x + j * (int)blockDim.x) + off;
        sum[j] = T(0);
        cnt[j] = 0;
        v[j] = T(0);
        r[j] = T(0);
        if (x < W) {
            const long i = rowi + x;
            if (x > 0) { sum[j] += phi[i - 1]; cnt[j]++; }
            if (y > 0) { sum[j] += phi[i - ld]; cnt[j]++; }
            if (x < W - 1) { sum[j] += phi[i + 1]; cnt[j]++; }
            if (y < H - 1) { sum[j] += phi[i + ld]; cnt[j]++; }
            v[j] = phi[i];
            r[j] = rhs[i];
        }
    }
    double m = 0.0;
#pragma unroll
    for (int j = 0; j < CELLS; j++) {
        const int x = 2 * (threadIdx.x + j * (int)blockDim.x) + off;
        if (x < W) {
            const T delta = omega_over_cnt<T>(a, cnt[j]) * (sum[j] - (T)cnt[j] * v[j] - r[j]);
            phi[rowi + x] = v[j] + delta;
            if (TRACK) {
                const double ad = fabs((double)delta);
                m = ad > m ? ad : m;
            }
        }
    }
    return m;
}

template <typename T, bool TRACK, int CELLS>
__global__ void __launch_bounds__(kStripeThreads, 2)
    k_stripe_a(T *__restrict__ phi, const T *__restrict__ rhs, Ctl *ctl, SolveArgs a, int R)
{
    if (vol_load(&ctl->halt)) return;
    const int y0 = blockIdx.x * R, y1 = min(y0 + R, a.H);
    double m = 0.0;
    // lines of one row (128 B each); threads [0, L) prefetch the next step's
    // new phi row, threads [L, 2L) its right-hand-side row
    const int L = (int)((a.W * sizeof(T) + 127) / 128);
    for (int j = 0; j <= y1 - y0; j++) {
        const int yr = y0 + j;
        const int t = threadIdx.x;
        if (yr + 2 < a.H && t < L) prefetch_l2(phi + (long)(yr + 2) * a.ld + t * (128 / sizeof(T)));
        else if (yr + 1 < y1 && t >= L && t < 2 * L)
            prefetch_l2(rhs + (long)(yr + 1) * a.ld + (t - L) * (128 / sizeof(T)));
        if (yr < y1) m = fmax(m, relax_row<T, TRACK, CELLS>(phi, rhs, a, yr, 0));
        __syncthreads();
        const int yb = yr - 1;
        if (yb >= y0 + 1 && yb <= y1 - 2) m = fmax(m, relax_row<T, TRACK, CELLS>(phi, rhs, a, yb, 1));
    }
    if (TRACK) {
        double v[1] = {m};
        block_reduce<1, 1u>(v);
        if (threadIdx.x == 0 && v[0] > 0.0) atomicMax(&ctl->maxbits, (unsigned long long)__double_as_longlong(v[0]));
    }
}

// Black cells of the first and last row of every stripe; the last block
// closes the sweep (end_of_sweep).  blockIdx.y = 2*stripe + {0: first, 1: last}.
template <typename T, bool TRACK, int CELLS>
__global__ void __launch_bounds__(kStripeThreads, 2)
    k_stripe_b(T *__restrict__ phi, const T *__restrict__ rhs, Ctl *ctl, SolveArgs a, int R)
{
    if (vol_load(&ctl->halt)) return;
    const int st = blockIdx.y >> 1, which = blockIdx.y & 1;
    const int y0 = st * R, y1 = min(y0 + R, a.H);
    const int y = which ? y1 - 1 : y0;
    double m = 0.0;
    if (!(which && y == y0)) m = relax_row<T, TRACK, CELLS>(phi, rhs, a, y, 1);
    if (TRACK) {
        double v[1] = {m};
        block_reduce<1, 1u>(v);
        m = v[0];
    }
    if (threadIdx.x == 0) {
        if (TRACK && m > 0.0) atomicMax(&ctl->maxbits, (unsigned long long)__double_as_longlong(m));
        __threadfence();
        const unsigned t = atomicAdd(&ctl->blocks_done, 1u);
        if (t == gridDim.x * gridDim.y - 1) {
            __threadfence();
            end_of_sweep(ctl, a);
        }
    }
}

// Rows per stripe such that all stripes are resident at once (one wave):
// stripes = resident blocks per SM x SMs.
inline int stripe_rows(int H, int resident)
{
    const int target = resident > 0 ? resident : 304;
    int R = (H + target - 1) / target;
    return R < 3 ? 3 : R;
}

#include "sor_stream.cuh"
#include "sor_stream2.cuh"

// Launch shape of the ping-pong stream sweep: G 4-cell groups per thread,
// T threads (one row of the grid per block), ns stripes of R rows; rows
// staged by bulk copies (tma, rows of wpad floats, smem bytes of dynamic
// shared memory) or loaded into registers.
struct StreamPlan {
    int G = 0, T = 0, R = 0, ns = 0;
    int tma = 0, wpad = 0;
    size_t smem = 0;
    int two = 0;          // two sweeps per pass (k_sweep2_tma) available
    size_t smem2 = 0;
};

int stream_plan(int dev, int W, int H, int ld, bool allow_tma, StreamPlan *p)
{
    const int groups = (W + 3) / 4;
    // two groups per thread at most: four would not fit in 128 registers
    if (H < 3 || ld % 4 != 0 || groups > 2 * kStreamThreadsMax) return PCD_BAD_ARG;
    const int G = groups <= kStreamThreadsMax ? 1 : 2;
    const int T = 32 * ceil_div(ceil_div(groups, G), 32);
    int sms = 0, bps = 0, max_smem = 0;
    PCD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    PCD_CUDA(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    const int wpad = 4 * groups;
    const size_t smem = tma_smem_bytes(wpad);
    const bool tma = allow_tma && smem <= (size_t)max_smem;
    if (tma) {
        const void *fns[2] = {G == 1 ? (const void *)k_sweep_tma<1, false> : (const void *)k_sweep_tma<2, false>,
                              G == 1 ? (const void *)k_sweep_tma<1, true> : (const void *)k_sweep_tma<2, true>};
        for (const void *fn : fns) PCD_CUDA(allow_shared(fn));
        int bps_t = 0;
        PCD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, fns[0], T, smem));
        PCD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps_t, fns[1], T, smem));
        bps = std::min(bps, bps_t);
    } else if (G == 1) {
        PCD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, k_sweep_stream<1, false>, T, 0));
    } else {
        PCD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, k_sweep_stream<2, false>, T, 0));
    }
    if (bps < 1) return PCD_BAD_ARG;
    int ns = std::min(bps * sms, ceil_div(H, kStreamRowsMin));
    if (ns < 1) ns = 1;
    // even stripe heights: every stripe starts on an even row (the two-sweep
    // pass relies on it for its compile-time cell parities)
    const int R = 2 * ceil_div(ceil_div(H, ns), 2);
    p->G = G;
    p->T = T;
    p->R = R;
    p->ns = ceil_div(H, R);
    p->tma = tma ? 1 : 0;
    p->wpad = wpad;
    p->smem = tma ? smem : 0;
    // the two-sweep pass: whole 4G-cell groups (W a multiple of 4G, one
    // group column per thread), one block per SM, stripes of >= 8 rows
    const size_t smem2 = tma2_smem_bytes(wpad, T);
    p->two = 0;
    p->smem2 = 0;
    if (tma && W % (4 * G) == 0 && T * 4 * G == W && smem2 + 1024 <= (size_t)max_smem && p->R >= 8 &&
        p->R % 2 == 0) {
        const void *fns2[2] = {G == 1 ? (const void *)k_sweep2_tma<1, false> : (const void *)k_sweep2_tma<2, false>,
                               G == 1 ? (const void *)k_sweep2_tma<1, true> : (const void *)k_sweep2_tma<2, true>};
        int ok2 = 1;
        for (const void *fn : fns2) {
            PCD_CUDA(allow_shared(fn));
            int b2 = 0;
            PCD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b2, fn, T, smem2));
            if (b2 < 1) ok2 = 0;
        }
        if (ok2) {
            p->two = 1;
            p->smem2 = smem2;
        }
    }
    return PCD_OK;
}

constexpr long kTmaSpinLimit = 1l << 22;

// Two sweeps from ein into eout (one when a single sweep is left before
// max_iter).
template <bool TRACK>
void launch_stream2_t(const StreamPlan &p, const float *ein, float *eout, const float *r, Ctl *ctl,
                      const SolveArgs &a, int out_idx, cudaStream_t s)
{
    if (p.G == 1)
        k_sweep2_tma<1, TRACK><<<p.ns, p.T, p.smem2, s>>>(ein, eout, r, ctl, a, p.R, out_idx, p.wpad, kTmaSpinLimit);
    else
        k_sweep2_tma<2, TRACK><<<p.ns, p.T, p.smem2, s>>>(ein, eout, r, ctl, a, p.R, out_idx, p.wpad, kTmaSpinLimit);
}

template <bool TRACK>
void launch_stream_t(const StreamPlan &p, const float *ein, float *eout, const float *r, Ctl *ctl, const SolveArgs &a,
                     int out_idx, cudaStream_t s)
{
    if (p.tma) {
        if (p.G == 1)
            k_sweep_tma<1, TRACK><<<p.ns, p.T, p.smem, s>>>(ein, eout, r, ctl, a, p.R, out_idx, p.wpad, kTmaSpinLimit);
        else
            k_sweep_tma<2, TRACK><<<p.ns, p.T, p.smem, s>>>(ein, eout, r, ctl, a, p.R, out_idx, p.wpad, kTmaSpinLimit);
    } else if (p.G == 1) {
        k_sweep_stream<1, TRACK><<<p.ns, p.T, 0, s>>>(ein, eout, r, ctl, a, p.R, out_idx);
    } else {
        k_sweep_stream<2, TRACK><<<p.ns, p.T, 0, s>>>(ein, eout, r, ctl, a, p.R, out_idx);
    }
}


__global__ void k_fill(double *p, int W, int H, int ld, double v)
{
    const long n = (long)W * H;
    for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x) {
        const int y = (int)(t / W), x = (int)(t - (long)y * W);
        p[(long)y * ld + x] = v;
    }
}

inline int grid_blocks(long n) { return (int)std::min<long>(kResidualBlocksMax, (n + kThreads - 1) / kThreads); }

}  // namespace

double resolve_omega(double omega, int W, int H)
{
    if (omega > 0.0) return omega;
    if (omega == 0.0) return 2.0 / (1.0 + 3.14159265 / W);  // solver.cpp:71
    const int n = W > H ? W : H;
    if (n < 2) return 1.0;
    const double mu = 0.5 * (1.0 + std::cos(M_PI / n));
    return 2.0 / (1.0 + std::sqrt(1.0 - mu * mu));
}

int SolverWorkspace::reserve(size_t n)
{
    if (!ctl) {
        PCD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        PCD_CUDA(cudaMalloc(&ctl, sizeof(Ctl)));
        PCD_CUDA(cudaMallocHost(&ctl_host, 2 * sizeof(Ctl)));
        PCD_CUDA(cudaMalloc(&partials, 3 * sizeof(double) * kResidualBlocksMax));
        max_partials = kResidualBlocksMax;
        for (int k = 0; k < 2; k++) PCD_CUDA(cudaEventCreateWithFlags(&ev[k], cudaEventDisableTiming));
        PCD_CUDA(cudaEventCreate(&t0));
        PCD_CUDA(cudaEventCreate(&t1));
        PCD_CUDA(cudaEventCreate(&k0));
        PCD_CUDA(cudaEventCreate(&k1));
    }
    if (n > cells) {
        if (mask) cudaFree(mask);
        if (e32) cudaFree(e32);
        if (e32b) cudaFree(e32b);
        if (r32) cudaFree(r32);
        if (r64) cudaFree(r64);
        mask = nullptr; e32 = nullptr; e32b = nullptr; r32 = nullptr; r64 = nullptr;
        cells = 0;  // (until all of them are there again)
        for (auto &kv : graphs) cudaGraphExecDestroy(kv.second.exec);
        graphs.clear();
        PCD_CUDA(cudaMalloc(&mask, n));
        PCD_CUDA(cudaMalloc(&e32, n * sizeof(float)));
        PCD_CUDA(cudaMalloc(&e32b, n * sizeof(float)));
        PCD_CUDA(cudaMalloc(&r32, n * sizeof(float)));
        PCD_CUDA(cudaMalloc(&r64, n * sizeof(double)));
        cells = n;
    }
    return PCD_OK;
}

void SolverWorkspace::release()
{
    for (auto &kv : graphs) cudaGraphExecDestroy(kv.second.exec);
    graphs.clear();
    if (mask) cudaFree(mask);
    if (e32) cudaFree(e32);
    if (e32b) cudaFree(e32b);
    if (r32) cudaFree(r32);
    if (r64) cudaFree(r64);
    if (xbuf) cudaFree(xbuf);
    if (flags) cudaFree(flags);
    if (part) cudaFree(part);
    if (bx) cudaFree(bx);
    if (rx) cudaFree(rx);
    r64 = nullptr; xbuf = nullptr; flags = nullptr; part = nullptr; bx = nullptr; rx = nullptr;
    xbuf_elems = 0; max_ctas = 0; bx_bytes = 0; rx_bytes = 0;
    plans.clear();
    if (partials) cudaFree(partials);
    if (ctl) cudaFree(ctl);
    if (ctl_host) cudaFreeHost(ctl_host);
    for (int k = 0; k < 2; k++)
        if (ev[k]) cudaEventDestroy(ev[k]);
    if (t0) cudaEventDestroy(t0);
    if (t1) cudaEventDestroy(t1);
    if (k0) cudaEventDestroy(k0);
    if (k1) cudaEventDestroy(k1);
    mask = nullptr; e32 = nullptr; e32b = nullptr; r32 = nullptr; partials = nullptr; ctl = nullptr;
    ctl_host = nullptr;
    cells = 0;
}

namespace {

template <typename T, bool TRACK, int CELLS>
void launch_stripes_c(T *phi, const T *rhs, Ctl *ctl, const SolveArgs &a, int R, int ns, dim3 gb, cudaStream_t s)
{
    k_stripe_a<T, TRACK, CELLS><<<ns, kStripeThreads, 0, s>>>(phi, rhs, ctl, a, R);
    k_stripe_b<T, TRACK, CELLS><<<gb, kStripeThreads, 0, s>>>(phi, rhs, ctl, a, R);
}

template <typename T, bool TRACK>
int launch_stripes(T *phi, const T *rhs, Ctl *ctl, const SolveArgs &a, int R, int ns, dim3 gb, int cells,
                   cudaStream_t s)
{
    if (cells <= 1) launch_stripes_c<T, TRACK, 1>(phi, rhs, ctl, a, R, ns, gb, s);
    else if (cells <= 2) launch_stripes_c<T, TRACK, 2>(phi, rhs, ctl, a, R, ns, gb, s);
    else if (cells <= 4) launch_stripes_c<T, TRACK, 4>(phi, rhs, ctl, a, R, ns, gb, s);
    else launch_stripes_c<T, TRACK, kRowCellsMax>(phi, rhs, ctl, a, R, ns, gb, s);
    return PCD_OK;
}

// Polls of a tagged word before a wait gives up: 0.21 us each, together about half a
// second (a withheld word ends a 256^2 solve after 21.6 ms with a limit of 100000).
constexpr long long kWordPolls = 1ll << 21;

// The tagged words' buffer, zeroed: tags start at 1 in every solve, and no word
// of an earlier one may match.
int reserve_words(SolverWorkspace &ws, size_t need, cudaStream_t s)
{
    if (need > ws.rx_bytes) {
        if (ws.rx) cudaFree(ws.rx);
        ws.rx = nullptr;
        ws.rx_bytes = 0;
        PCD_CUDA(cudaMalloc(&ws.rx, need));
        ws.rx_bytes = need;
    }
    PCD_CUDA(cudaMemsetAsync(ws.rx, 0, need, s));
    return PCD_OK;
}

// The FP64 refresh of a single solve: the potential alternates between phi and
// the workspace's r64.
RefreshJob refresh_job(const SolverWorkspace &ws, const double *b, double *phi, const SolveArgs &a)
{
    RefreshJob j{};
    j.b = b;
    j.phi = phi;
    j.phi2 = ws.r64;
    j.e0 = ws.e32;
    j.e1 = ws.e32b;
    j.r32 = ws.r32;
    j.ctl = ws.ctl;
    j.error = &ws.ctl->error;
    j.partials = ws.partials;
    j.W = a.W;
    j.H = a.H;
    j.ld = a.ld;
    j.nblk = refresh_shape(a.W, a.H, a.ld, kResidualBlocksMax, ws.sms, &j.rows);
    return j;
}

// Enqueues one chunk of `sweeps` sweeps (plus the checks that follow them) on s.
template <bool MASKED>
int enqueue_chunk(SolverWorkspace &ws, const double *b, double *phi, const SolveArgs &a, int precision,
                  int sweeps, cudaStream_t s, int *nodes, int sched, const StreamPlan &sp)
{
    const bool stripes = sched == PCD_SCHED_STRIPES;
    const int half = (a.W + 1) >> 1;
    const int blocks = ceil_div((long)a.H * half, kThreads);
    const int rblocks = grid_blocks((long)a.W * a.H);
    const bool track = (a.stop == PCD_STOP_MAX_UPDATE);
    int n = 0;
    if (!MASKED && stripes) {
        const int R = stripe_rows(a.H, ws.stripe_resident);
        const int ns = (a.H + R - 1) / R;
        const dim3 gb(1, 2 * ns);  // one block per boundary row (relax_row strides over the row)
        const int cells = ceil_div(half, kStripeThreads);
        for (int k = 0; k < sweeps; k++) {
            if (precision == PCD_PREC_MIXED) {
                if (track) PCD_TRY((launch_stripes<float, true>(ws.e32, ws.r32, ws.ctl, a, R, ns, gb, cells, s)));
                else PCD_TRY((launch_stripes<float, false>(ws.e32, ws.r32, ws.ctl, a, R, ns, gb, cells, s)));
            } else {
                if (track) PCD_TRY((launch_stripes<double, true>(phi, b, ws.ctl, a, R, ns, gb, cells, s)));
                else PCD_TRY((launch_stripes<double, false>(phi, b, ws.ctl, a, R, ns, gb, cells, s)));
            }
            n += 2;
        }
        sweeps = 0;
    }
    if (!MASKED && sched == PCD_SCHED_STREAM) {
        // launch k reads buffer k&1 and writes the other (two sweeps per
        // launch where the plan allows, a single sweep for an odd rest); the
        // settle kernel moves the latest correction into e32 for the refinement
        int k = 0;
        for (int done = 0; done < sweeps; k++) {
            const float *ein = (k & 1) ? ws.e32b : ws.e32;
            float *eout = (k & 1) ? ws.e32 : ws.e32b;
            const int out = (k & 1) ? 0 : 1;
            if (sp.two && sweeps - done >= 2) {
                if (track) launch_stream2_t<true>(sp, ein, eout, ws.r32, ws.ctl, a, out, s);
                else launch_stream2_t<false>(sp, ein, eout, ws.r32, ws.ctl, a, out, s);
                done += 2;
            } else {
                if (track) launch_stream_t<true>(sp, ein, eout, ws.r32, ws.ctl, a, out, s);
                else launch_stream_t<false>(sp, ein, eout, ws.r32, ws.ctl, a, out, s);
                done += 1;
            }
            n++;
        }
        k_stream_settle<<<rblocks, kThreads, 0, s>>>(ws.e32, ws.e32b, ws.ctl, a);
        n++;
        sweeps = 0;
    }
    for (int k = 0; k < sweeps; k++) {
        for (int color = 0; color < 2; color++) {
            const int last = color == 1;
            if (precision == PCD_PREC_MIXED) {
                if (track)
                    k_rb_half<float, MASKED, true><<<blocks, kThreads, 0, s>>>(ws.e32, ws.r32, ws.mask, ws.ctl, a, color, last);
                else
                    k_rb_half<float, MASKED, false><<<blocks, kThreads, 0, s>>>(ws.e32, ws.r32, ws.mask, ws.ctl, a, color, last);
            } else {
                if (track)
                    k_rb_half<double, MASKED, true><<<blocks, kThreads, 0, s>>>(phi, b, ws.mask, ws.ctl, a, color, last);
                else
                    k_rb_half<double, MASKED, false><<<blocks, kThreads, 0, s>>>(phi, b, ws.mask, ws.ctl, a, color, last);
            }
            n++;
        }
    }
    if (precision == PCD_PREC_MIXED) {
        k_refine_residual<MASKED><<<rblocks, kThreads, 0, s>>>(phi, ws.e32, b, ws.mask, ws.r32, ws.ctl, ws.partials, a, 0);
        k_refine_update<<<rblocks, kThreads, 0, s>>>(phi, ws.e32, ws.ctl, a);
        n += 2;
    } else if (a.stop == PCD_STOP_REL_RESIDUAL) {
        k_residual64<MASKED><<<rblocks, kThreads, 0, s>>>(phi, b, ws.mask, ws.ctl, ws.partials, a, 1, 0, 1);
        n++;
    }
    PCD_CUDA(cudaGetLastError());
    *nodes = n;
    return PCD_OK;
}

// Smallest grid (cells) that AUTO hands to the tile passes rather than the
// persistent schedule (the smallest size measured: 64^2, where the tile
// passes took 1.0 ms against 2.2 ms to the reference's stop at 1e-7).
constexpr long kTileMinCells = 64L * 64L;

int get_chunk_graph(SolverWorkspace &ws, const double *b, double *phi, const SolveArgs &a, int precision,
                    int masked, int sweeps, cudaStream_t s, SolverWorkspace::GraphEntry **out, int sched,
                    const StreamPlan &sp)
{
    std::vector<long long> key = {(long long)(uintptr_t)b, (long long)(uintptr_t)phi, a.W, a.H, a.ld, a.stop,
                                  a.max_iter, precision, masked, sweeps, sched, sp.G, sp.T, sp.R, sp.tma, sp.two};
    long long tb, ob;
    std::memcpy(&tb, &a.tol, 8);
    std::memcpy(&ob, &a.omega, 8);
    key.push_back(tb);
    key.push_back(ob);
    auto it = ws.graphs.find(key);
    if (it != ws.graphs.end()) {
        *out = &it->second;
        return PCD_OK;
    }
    cudaGraph_t g;
    int nodes = 0;
    PCD_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    int st = masked ? enqueue_chunk<true>(ws, b, phi, a, precision, sweeps, s, &nodes, PCD_SCHED_LAUNCHES, sp)
                    : enqueue_chunk<false>(ws, b, phi, a, precision, sweeps, s, &nodes, sched, sp);
    cudaError_t ce = cudaStreamEndCapture(s, &g);
    if (st != PCD_OK) {
        if (ce == cudaSuccess) cudaGraphDestroy(g);
        return st;
    }
    if (ce != cudaSuccess) {
        set_error(std::string("cudaStreamEndCapture: ") + cudaGetErrorString(ce));
        return PCD_DEVICE_ERROR;
    }
    cudaGraphExec_t exec;
    ce = cudaGraphInstantiate(&exec, g, 0);
    cudaGraphDestroy(g);
    if (ce != cudaSuccess) {
        set_error(std::string("cudaGraphInstantiate: ") + cudaGetErrorString(ce));
        return PCD_DEVICE_ERROR;
    }
    if (ws.graphs.size() > 64) {
        for (auto &kv : ws.graphs) cudaGraphExecDestroy(kv.second.exec);
        ws.graphs.clear();
    }
    auto &e = ws.graphs[key];
    e.exec = exec;
    e.nodes = nodes;
    *out = &e;
    return PCD_OK;
}

}  // namespace

namespace {

template <typename Plan, typename Make>
int cached_plan(SolverWorkspace &ws, std::vector<int> key, Plan *out, Make make)
{
    // entry: status byte, then the plan
    auto it = ws.plans.find(key);
    if (it == ws.plans.end()) {
        Plan p{};
        const int st = make(&p);
        if (st != PCD_OK && st != PCD_BAD_ARG) return st;
        if (ws.plans.size() >= 256) ws.plans.clear();
        std::vector<char> v(1 + sizeof(Plan));
        v[0] = (char)st;
        std::memcpy(v.data() + 1, &p, sizeof(Plan));
        it = ws.plans.emplace(std::move(key), std::move(v)).first;
    }
    std::memcpy(out, it->second.data() + 1, sizeof(Plan));
    return it->second[0];
}

enum { kPlanResident, kPlanCluster, kPlanTile, kPlanPersist, kPlanBlocks, kPlanBlocks64 };


// One cooperative launch per solve (sor_persist.cu), bracketed by the FP64
// residual kernels that supply ||b|| / r64 before and the exact statistics after.
int solve_persistent(SolverWorkspace &ws, const double *b, double *phi, const SolveArgs &a, int precision,
                     const pcd_solve_opts &o, int G, size_t smem, pcd_solve_stats *stats, cudaStream_t s)
{
    const bool mixed = precision == PCD_PREC_MIXED;
    const size_t xe = (size_t)G * 4 * a.W;
    if (xe > ws.xbuf_elems) {
        if (ws.xbuf) cudaFree(ws.xbuf);
        ws.xbuf = nullptr;
        ws.xbuf_elems = 0;
        PCD_CUDA(cudaMalloc(&ws.xbuf, xe * sizeof(double)));
        ws.xbuf_elems = xe;
    }
    if (G > ws.max_ctas) {
        if (ws.flags) cudaFree(ws.flags);
        if (ws.part) cudaFree(ws.part);
        ws.flags = nullptr;
        ws.part = nullptr;
        ws.max_ctas = 0;
        PCD_CUDA(cudaMalloc(&ws.flags, (G + 1) * sizeof(unsigned)));
        PCD_CUDA(cudaMalloc(&ws.part, 2 * 3 * G * sizeof(double)));
        ws.max_ctas = G;
    }
    PCD_CUDA(cudaMemsetAsync(ws.flags, 0, (G + 1) * sizeof(unsigned), s));

    PersistArgs pa{};
    pa.W = a.W; pa.H = a.H; pa.ld = a.ld; pa.G = G;
    pa.b = b; pa.phi = phi; pa.r64 = ws.r64;
    pa.xbuf = ws.xbuf; pa.flags = ws.flags; pa.bar = ws.flags + G; pa.part = ws.part; pa.ctl = ws.ctl;
    pa.stop = a.stop; pa.max_iter = a.max_iter; pa.tol = a.tol;
    if (o.check_every > 0) pa.check_every = o.check_every;
    else if (a.stop == PCD_STOP_MAX_UPDATE) pa.check_every = mixed ? 16 : 8;
    else pa.check_every = 32;
    if (mixed && o.refine_every > 0 && o.refine_every < pa.check_every) pa.check_every = o.refine_every;
    for (int c = 0; c < 5; c++) { pa.w64[c] = a.w64[c]; pa.w32[c] = a.w32[c]; }
    pa.spin_limit = ws.wait_limit > 0 ? ws.wait_limit : 1ll << 24;
    pa.withhold = ws.withhold_flag;
    PCD_CUDA(cudaEventRecord(ws.k0, s));
    PCD_TRY(launch_persist(pa, mixed, smem, s));
    PCD_CUDA(cudaEventRecord(ws.k1, s));

    // exact FP64 statistics of the returned phi
    const int rblocks = grid_blocks((long)a.W * a.H);
    k_residual64<false><<<rblocks, kThreads, 0, s>>>(phi, b, ws.mask, ws.ctl, ws.partials, a, 0, 1, 0);
    PCD_LAUNCHED(1);
    PCD_CUDA(cudaEventRecord(ws.t1, s));
    PCD_CUDA(cudaMemcpyAsync(&ws.ctl_host[0], ws.ctl, sizeof(Ctl), cudaMemcpyDeviceToHost, s));
    PCD_CUDA(cudaStreamSynchronize(s));
    const Ctl &c = ws.ctl_host[0];
    if (c.error) {
        set_error("persistent SOR: a bounded device wait gave up (status " + std::to_string(c.error) + ")");
        return c.error;
    }
    int converged = c.converged;
    if (a.stop == PCD_STOP_REL_RESIDUAL) converged = c.rel <= a.tol;
    if (stats) {
        stats->sweeps = c.sweeps;
        stats->converged = converged;
        stats->rel_residual = c.rel;
        stats->max_residual = c.rmax;
        stats->last_max_update = c.last_max;
        stats->residual_checks = c.checks + 2;
        float ms = 0.f;
        cudaEventElapsedTime(&ms, ws.t0, ws.t1);
        stats->device_ms = ms;
        cudaEventElapsedTime(&ms, ws.k0, ws.k1);
        stats->sweep_ms = ms;
        stats->schedule_used = PCD_SCHED_PERSISTENT;
    }
    return converged ? PCD_OK : PCD_NOT_CONVERGED;
}

// The CTA-count dependent buffers of the persistent schedules: G epoch flags
// plus a barrier counter, and 2 x G x 3 check partials.
int reserve_ctas(SolverWorkspace &ws, int G)
{
    if (G > ws.max_ctas) {
        if (ws.flags) cudaFree(ws.flags);
        if (ws.part) cudaFree(ws.part);
        ws.flags = nullptr;
        ws.part = nullptr;
        ws.max_ctas = 0;
        PCD_CUDA(cudaMalloc(&ws.flags, (G + 1) * sizeof(unsigned)));
        PCD_CUDA(cudaMalloc(&ws.part, 2 * 3 * G * sizeof(double)));
        ws.max_ctas = G;
    }
    return PCD_OK;
}

// Sweeps between the stop tests of the block schedule: a test costs an all-to-
// all exchange of partials (a few L2 round trips), so every 16 sweeps for the
// max-update stop and 32 for the relative residual, a multiple of the plan's
// sweeps per exchange.
int blocks_check_every(const SolveArgs &a, const pcd_solve_opts &o, const BlocksPlan &bp)
{
    const int ce = o.check_every > 0 ? o.check_every : (a.stop == PCD_STOP_MAX_UPDATE ? 16 : 32);
    return std::max(bp.K, (ce + bp.K - 1) / bp.K * bp.K);
}

// The end of a block solve: the exact FP64 statistics of the returned phi.
int finish_blocks(SolverWorkspace &ws, const double *b, const double *phi, const SolveArgs &a, int ce,
                  pcd_solve_stats *stats, cudaStream_t s)
{
    // exact FP64 statistics of the returned phi
    const int rblocks = grid_blocks((long)a.W * a.H);
    k_residual64<false><<<rblocks, kThreads, 0, s>>>(phi, b, ws.mask, ws.ctl, ws.partials, a, 0, 1, 0);
    PCD_LAUNCHED(1);
    PCD_CUDA(cudaEventRecord(ws.t1, s));
    PCD_CUDA(cudaMemcpyAsync(&ws.ctl_host[0], ws.ctl, sizeof(Ctl), cudaMemcpyDeviceToHost, s));
    PCD_CUDA(cudaStreamSynchronize(s));
    const Ctl &c = ws.ctl_host[0];
    if (c.error) {
        set_error("block SOR: a bounded device wait gave up (status " + std::to_string(c.error) + ")");
        return c.error;
    }
    int converged = c.converged;
    if (a.stop == PCD_STOP_REL_RESIDUAL) converged = c.rel <= a.tol;
    if (stats) {
        stats->sweeps = c.sweeps;
        stats->converged = converged;
        stats->rel_residual = c.rel;
        stats->max_residual = c.rmax;
        stats->last_max_update = c.last_max;
        stats->residual_checks = c.checks + 2;
        float ms = 0.f;
        cudaEventElapsedTime(&ms, ws.t0, ws.t1);
        stats->device_ms = ms;
        cudaEventElapsedTime(&ms, ws.k0, ws.k1);
        stats->sweep_ms = ms;
        stats->schedule_used = PCD_SCHED_BLOCKS;
        stats->check_every_used = ce;
    }
    return converged ? PCD_OK : PCD_NOT_CONVERGED;
}

// One cooperative launch per solve on 2-D blocks with deep halos
// (sor_blocks.cu), then the exact FP64 statistics of the returned phi.
int solve_blocks(SolverWorkspace &ws, const double *b, double *phi, const SolveArgs &a, const pcd_solve_opts &o,
                 const BlocksPlan &bp, pcd_solve_stats *stats, cudaStream_t s)
{
    const int G = bp.TY * bp.TX;
    const int xs = (a.W + 3) & ~3;
    const size_t need = 3 * (size_t)a.H * xs * sizeof(float);
    if (need > ws.bx_bytes) {
        if (ws.bx) cudaFree(ws.bx);
        ws.bx = nullptr;
        ws.bx_bytes = 0;
        PCD_CUDA(cudaMalloc(&ws.bx, need));
        ws.bx_bytes = need;
    }
    PCD_TRY(reserve_ctas(ws, G));
    PCD_CUDA(cudaMemsetAsync(ws.flags, 0, (G + 1) * sizeof(unsigned), s));

    BlocksArgs ba{};
    ba.W = a.W; ba.H = a.H; ba.ld = a.ld;
    ba.TY = bp.TY; ba.TX = bp.TX; ba.G = G; ba.K = bp.K; ba.RTmax = bp.RTmax; ba.xs = xs;
    ba.phi = phi; ba.r64 = ws.r64;
    ba.xb = static_cast<float *>(ws.bx);
    ba.r32x = static_cast<float *>(ws.bx) + 2 * (size_t)a.H * xs;
    ba.flags = ws.flags; ba.part = ws.part; ba.ctl = ws.ctl;
    ba.stop = a.stop; ba.max_iter = a.max_iter; ba.tol = a.tol;
    const int ce = blocks_check_every(a, o, bp);
    ba.check_every = ce;
    ba.cycle_cap = o.refine_every > 0 ? o.refine_every : 2048;
    ba.drop = o.refine_drop > 0.0 ? o.refine_drop : 3e-2;
    for (int c = 0; c < 5; c++) ba.w32[c] = a.w32[c];
    ba.spin_limit = ws.wait_limit > 0 ? ws.wait_limit : 1ll << 24;
    ba.withhold = ws.withhold_flag;
    PCD_CUDA(cudaEventRecord(ws.k0, s));
    PCD_TRY(launch_blocks(ba, bp.smem, s));
    PCD_CUDA(cudaEventRecord(ws.k1, s));

    return finish_blocks(ws, b, phi, a, ce, stats, s);
}

// The FP64 form (sor_blocks64.cu), on grids that bp, the layout of the rule
// below, fits; bp also fixes the stop tests' spacing.
int solve_blocks64(SolverWorkspace &ws, const double *b, double *phi, const SolveArgs &a, const pcd_solve_opts &o,
                   const BlocksPlan &bp, pcd_solve_stats *stats, cudaStream_t s)
{
    Blocks64Plan plan;
    const int st = cached_plan(ws, {kPlanBlocks64, a.W, a.H, o.block_sweeps}, &plan, [&](Blocks64Plan *p) {
        return blocks64_plan(ws.dev, a.W, a.H, o.block_sweeps, p);
    });
    if (st != PCD_OK) {
        if (st == PCD_BAD_ARG) set_error("block SOR: no FP64 layout for this grid");
        return st;
    }
    const size_t part_at = plan.xb_bytes, need = part_at + (size_t)2 * plan.TY * plan.TX * 32;
    PCD_TRY(reserve_words(ws, need, s));
    Blocks64Args ba{};
    ba.W = a.W; ba.H = a.H; ba.ld = a.ld;
    ba.b = b; ba.phi = phi;
    ba.xb = ws.rx;
    ba.part = static_cast<char *>(ws.rx) + part_at;
    ba.ctl = ws.ctl;
    ba.stop = a.stop; ba.max_iter = a.max_iter; ba.tol = a.tol; ba.omega = a.omega;
    const int ce = blocks_check_every(a, o, bp);
    ba.check_every = ce;
    for (int c = 0; c < 5; c++) ba.w64[c] = a.w64[c];
    ba.spin_limit = ws.wait_limit > 0 ? ws.wait_limit : kWordPolls;
    ba.withhold = ws.withhold_flag;
    PCD_CUDA(cudaEventRecord(ws.k0, s));
    PCD_TRY(launch_blocks64(ba, plan, s));
    PCD_CUDA(cudaEventRecord(ws.k1, s));
    return finish_blocks(ws, b, phi, a, ce, stats, s);
}

}  // namespace

namespace {

// Mixed precision on one cluster: cycles of [FP32 cluster sweeps, FP64
// residual refresh, phi += e] until the FP64 relative residual passes.  The
// next cycle is launched before the previous one's control block is read; a
// cycle launched after convergence returns at once.
int solve_cluster(SolverWorkspace &ws, const double *b, double *phi, const SolveArgs &a, const pcd_solve_opts &o,
                  const ClusterPlan &plan, pcd_solve_stats *stats, cudaStream_t s)
{
    const int rblocks = grid_blocks((long)a.W * a.H);
    // (r32 and the norms of the initial guess are the start's)
    PCD_CUDA(cudaMemsetAsync(ws.e32, 0, sizeof(float) * (size_t)a.H * a.ld, s));

    ClusterArgs ca{};
    ca.W = a.W; ca.H = a.H; ca.ld = a.ld; ca.khp = plan.khp;
    ca.e = ws.e32; ca.r32 = ws.r32; ca.ctl = ws.ctl;
    ca.check_every = o.check_every > 0 ? o.check_every : 16;
    ca.cycle_cap = o.refine_every > 0 ? o.refine_every : 2048;
    ca.max_iter = a.max_iter;
    ca.tol = a.tol;
    ca.drop = o.refine_drop > 0.0 ? o.refine_drop : 3e-2;
    for (int c = 0; c < 5; c++) ca.w32[c] = a.w32[c];
    ca.one_minus_omega = (float)(1.0 - a.omega);
    ca.depth = plan.depth;

    PCD_CUDA(cudaEventRecord(ws.k0, s));
    long launched = 0;
    const long max_cycles = (long)a.max_iter + 4;
    bool finished = false;
    while (!finished) {
        if (launched >= max_cycles) {
            set_error("cluster SOR: cycle budget exceeded without a done flag");
            return PCD_TIMEOUT;
        }
        PCD_TRY(launch_cluster(ca, plan, s));
        k_refine_residual<false><<<rblocks, kThreads, 0, s>>>(phi, ws.e32, b, ws.mask, ws.r32, ws.ctl, ws.partials, a, 0);
        PCD_LAUNCHED(1);
        k_refine_update<<<rblocks, kThreads, 0, s>>>(phi, ws.e32, ws.ctl, a);
        PCD_LAUNCHED(1);
        const int slot = (int)(launched & 1);
        PCD_CUDA(cudaMemcpyAsync(&ws.ctl_host[slot], ws.ctl, sizeof(Ctl), cudaMemcpyDeviceToHost, s));
        PCD_CUDA(cudaEventRecord(ws.ev[slot], s));
        launched++;
        if (launched >= 2) {
            const int prev = (int)((launched - 2) & 1);
            PCD_CUDA(cudaEventSynchronize(ws.ev[prev]));
            if (ws.ctl_host[prev].done) finished = true;
        }
    }
    PCD_CUDA(cudaEventRecord(ws.k1, s));
    PCD_CUDA(cudaEventRecord(ws.t1, s));
    PCD_CUDA(cudaMemcpyAsync(&ws.ctl_host[0], ws.ctl, sizeof(Ctl), cudaMemcpyDeviceToHost, s));
    PCD_CUDA(cudaStreamSynchronize(s));
    const Ctl &c = ws.ctl_host[0];
    if (stats) {
        stats->sweeps = c.sweeps;
        stats->converged = c.converged;
        stats->rel_residual = c.rel;
        stats->max_residual = c.rmax;
        stats->last_max_update = 0.0;
        stats->residual_checks = c.checks;
        float ms = 0.f;
        cudaEventElapsedTime(&ms, ws.t0, ws.t1);
        stats->device_ms = ms;
        cudaEventElapsedTime(&ms, ws.k0, ws.k1);
        stats->sweep_ms = ms;
        stats->schedule_used = PCD_SCHED_CLUSTER;
    }
    return c.converged ? PCD_OK : PCD_NOT_CONVERGED;
}

}  // namespace

namespace {

// How the resident sweeps end their launches, so that every grid keeps the
// stop tests (and with them the sweep counts) of the schedule it is resident
// for: the cluster's residual-estimate cycles, the tile passes' chunks with a
// test after every pass, or the persistent bands' chunks.
struct ResidentRule {
    int cycle = 0;               // 1: estimate cycles
    int dep = 1, lag = 0;        // cycle: estimates on multiples of dep, end lag sweeps later
    int chunk = 0, gran = 0;     // chunk: sweeps per launch, tracked every gran sweeps
    int sched = PCD_SCHED_TILES; // what the solve reports
};

// Grids that the tile passes take under any schedule.  Others (AUTO alone) keep
// the stop tests of the schedules that they had before.
bool tile_grid(int W, int ld) { return W >= 8 && W % 8 == 0 && ld % 4 == 0 && ld < kRefreshLdMax; }

// Most sweeps of a launch of tile passes (their counts of passes are rounded up in 32
// bits); no solve comes near it.
constexpr int kChunkSweepsMax = 1 << 30;

// FP32 sweeps between FP64 refreshes of the chunked mixed schedules.
int mixed_chunk(const SolveArgs &a, const pcd_solve_opts &o)
{
    const int n = std::max(a.W, a.H);
    int chunk;
    if (a.stop == PCD_STOP_MAX_UPDATE)
        // (the stop test runs after every pass either way)
        chunk = o.refine_every > 0 ? o.refine_every : std::max(32, std::min(128, n / 32));
    else
        // the FP64 refresh costs several FP32 sweeps; FP32 can carry ~2 digits
        // of the correction, i.e. hundreds of sweeps on large grids
        chunk = o.refine_every > 0 ? o.refine_every
                                   : (o.check_every > 0 ? o.check_every : std::max(32, std::min(256, n / 16)));
    if (chunk > a.max_iter && a.max_iter > 0) chunk = a.max_iter;
    return chunk;
}

// Whether (and under which rule) the mixed solve's sweeps run resident.
int resident_rule(SolverWorkspace &ws, const SolveArgs &a, const pcd_solve_opts &o, ResidentPlan *plan,
                  ResidentRule *rule)
{
    if (o.precision != PCD_PREC_MIXED || o.schedule != PCD_SCHED_AUTO || a.ld >= kRefreshLdMax) return PCD_BAD_ARG;
    const int W = a.W, H = a.H;
    int st = cached_plan(ws, {kPlanResident, W, H}, plan, [&](ResidentPlan *p) { return resident_plan(ws.dev, W, H, p); });
    if (st != PCD_OK) return st;
    ResidentRule r;
    if (a.stop == PCD_STOP_REL_RESIDUAL) {
        ClusterPlan cp{};
        st = cached_plan(ws, {kPlanCluster, W, H}, &cp, [&](ClusterPlan *p) { return cluster_plan(ws.dev, W, H, 4, p); });
        if (st == PCD_OK) {
            r.cycle = 1;
            r.dep = std::max(1, cp.depth);
            r.lag = cp.rr_l ? cp.depth : 0;
            *rule = r;
            return PCD_OK;
        }
        if (st != PCD_BAD_ARG) return st;
    }
    const int depth = o.check_every > 0 && o.check_every <= 2 ? 2 : 4;
    TilePlan tp{};
    st = tile_grid(W, a.ld) ? cached_plan(ws, {kPlanTile, W, H, depth}, &tp,
                                          [&](TilePlan *p) { return tile_plan(ws.dev, W, H, depth, p); })
                            : PCD_BAD_ARG;
    if (st != PCD_OK && st != PCD_BAD_ARG) return st;
    if (st == PCD_OK && (long)W * H >= kTileMinCells) {
        r.chunk = mixed_chunk(a, o);
        r.gran = o.check_every > 0 ? std::min(o.check_every, 4) : 4;
    } else {
        struct { int G; size_t smem; } pp{};
        st = cached_plan(ws, {kPlanPersist, W, H}, &pp,
                         [&](decltype(pp) *p) { return persist_grid(ws.dev, W, H, true, &p->G, &p->smem); });
        if (st != PCD_OK) return st;
        r.chunk = o.check_every > 0 ? o.check_every : (a.stop == PCD_STOP_MAX_UPDATE ? 16 : 32);
        if (o.refine_every > 0 && o.refine_every < r.chunk) r.chunk = o.refine_every;
        r.gran = r.chunk;
    }
    if (a.stop != PCD_STOP_MAX_UPDATE) r.gran = 0;
    if (r.gran > 0 && (r.chunk - 1) / r.gran + 1 > kResidentChecksMax) return PCD_BAD_ARG;
    *rule = r;
    return PCD_OK;
}

// A mixed-precision solve's chunks: launch(): one chunk of FP32 sweeps; after each
// the FP64 refresh.  Chunk i + 1 is launched before chunk i's control block is
// inspected, and does nothing but bring the potential home where the solve is
// done.  The refresh leaves the control block in host memory itself: a copy
// between it and the next chunk's launch took 9 us.
template <typename Launch>
int run_chunks(SolverWorkspace &ws, RefreshJob job, const SolveArgs &a, long max_launches, int sched, int form,
               const char *what, pcd_solve_stats *stats, int *nans, cudaStream_t s, Launch launch)
{
    PCD_CUDA(cudaEventRecord(ws.k0, s));
    const Ctl *last = nullptr;
    for (long launched = 0; !last; launched++) {
        if (launched >= max_launches) {
            set_error(std::string(what) + ": launch budget exceeded without a done flag");
            return PCD_TIMEOUT;
        }
        PCD_TRY(launch());
        const int slot = (int)(launched & 1);
        job.report = &ws.ctl_host[slot];
        PCD_TRY(launch_refresh(nullptr, job, 1, job.nblk, a.stop == PCD_STOP_REL_RESIDUAL ? a.tol : -1.0, s));
        PCD_CUDA(cudaEventRecord(ws.ev[slot], s));
        if (launched < 1) continue;
        PCD_CUDA(cudaEventSynchronize(ws.ev[slot ^ 1]));
        const Ctl &c = ws.ctl_host[slot ^ 1];
        if (c.done || c.error || c.nan_cells) last = &c;
    }
    PCD_CUDA(cudaEventRecord(ws.k1, s));
    PCD_CUDA(cudaEventRecord(ws.t1, s));
    PCD_CUDA(cudaStreamSynchronize(s));
    const Ctl &c = *last;
    *nans = c.nan_cells;
    if (c.error) {
        set_error(std::string(what) + ": a bounded device wait gave up (status " + std::to_string(c.error) + ")");
        return c.error;
    }
    if (stats) {
        stats->sweeps = c.sweeps;
        stats->converged = c.converged;
        stats->rel_residual = c.rel;
        stats->max_residual = c.rmax;
        stats->last_max_update = c.last_max;
        stats->residual_checks = c.checks;
        float ms = 0.f;
        cudaEventElapsedTime(&ms, ws.t0, ws.t1);
        stats->device_ms = ms;
        cudaEventElapsedTime(&ms, ws.k0, ws.k1);
        stats->sweep_ms = ms;
        stats->schedule_used = sched;
        stats->sweep_form = form;
    }
    return c.converged ? PCD_OK : PCD_NOT_CONVERGED;
}

// Mixed precision on resident tiles: launches of [FP32 sweeps, FP64 residual
// refresh, phi += e] until the stop test passes.  The next launch is enqueued
// before the previous one's control block is read; a launch after the stop
// returns at once.  The NaN count of b is read with the first control block:
// where there are any nothing has been done (*nans tells the caller).
int solve_resident(SolverWorkspace &ws, const double *b, double *phi, const SolveArgs &a, const pcd_solve_opts &o,
                   const ResidentPlan &plan, const ResidentRule &rule, pcd_solve_stats *stats, int *nans,
                   cudaStream_t s)
{
    const int G = plan.TX * plan.TY;
    const size_t part_at = plan.xb_bytes, gmax_at = part_at + 2 * (size_t)G * sizeof(unsigned long long);
    const size_t bar_at = gmax_at + kResidentChecksMax * sizeof(unsigned), need = bar_at + 64;
    PCD_TRY(reserve_words(ws, need, s));

    ResidentArgs ra{};
    ra.W = a.W; ra.H = a.H;
    ra.e = ws.e32; ra.r32 = ws.r32; ra.ctl = ws.ctl;
    char *rx = static_cast<char *>(ws.rx);
    ra.xb = rx;
    ra.part = reinterpret_cast<unsigned long long *>(rx + part_at);
    ra.gmax = reinterpret_cast<unsigned *>(rx + gmax_at);
    ra.bar = reinterpret_cast<unsigned *>(rx + bar_at);
    ra.max_iter = a.max_iter;
    ra.cycle = rule.cycle;
    ra.nsw = rule.cycle ? (o.refine_every > 0 ? o.refine_every : 2048) : rule.chunk;
    // (the kernel adds it to a sweep count: up to 2^30, beyond any launch's sweeps)
    ra.check_every = o.check_every > 0 ? std::min(o.check_every, 1 << 30) : 16;
    ra.dep = rule.dep;
    ra.lag = rule.lag;
    ra.gran = rule.gran;
    ra.tol = a.tol;
    ra.drop = o.refine_drop > 0.0 ? o.refine_drop : 3e-2;
    for (int c = 0; c < 5; c++) ra.w32[c] = a.w32[c];
    ra.spin_limit = ws.wait_limit > 0 ? ws.wait_limit : kWordPolls;
    ra.withhold = ws.withhold_flag;

    const long max_launches = rule.cycle ? (long)a.max_iter + 4 : (long)a.max_iter / std::max(1, rule.chunk) + 3;
    return run_chunks(ws, refresh_job(ws, b, phi, a), a, max_launches, rule.sched, 1, "resident SOR", stats, nans, s,
                      [&] { return launch_resident(ra, plan, s); });
}

// Tile passes over a grid in HBM (sor_tile.cu), nsw sweeps a pass; the update of a
// pass's last sweep is tested by the max-update stop, for each pass or for a chunk's
// last.
int solve_tiles(SolverWorkspace &ws, const double *b, double *phi, const SolveArgs &a, const TilePlan &plan, int nsw,
                int chunk, bool each, int sched, pcd_solve_stats *stats, cudaStream_t s)
{
    chunk = std::min(chunk, kChunkSweepsMax);
    // a word a tile, and for the max-update stop one a pass
    const size_t tiles = (size_t)plan.ncol * plan.nrow, passes = (size_t)(chunk - 1) / nsw + 1;
    PCD_TRY(reserve_words(ws, sizeof(unsigned) * (tiles + (a.stop == PCD_STOP_MAX_UPDATE ? passes : 0)), s));
    unsigned *done = static_cast<unsigned *>(ws.rx);
    TileMaps maps;
    PCD_TRY(tile_maps(ws.e32, ws.e32b, ws.r32, a.W, a.H, plan.ncol, plan.rows, 2 * plan.K, &maps));
    int nans = 0;
    return run_chunks(ws, refresh_job(ws, b, phi, a), a, (long)a.max_iter / chunk + 3, sched, 2, "tile SOR",
                      stats, &nans, s, [&] {
                          return launch_tile(plan, maps, ws.ctl, done, done + tiles, a, nsw, chunk, each,
                                             ws.wait_limit > 0 ? ws.wait_limit : kWordPolls, ws.withhold_flag, s);
                      });
}

}  // namespace

int residual_rel(SolverWorkspace &ws, const double *b, const double *phi, int W, int H, int ld, cudaStream_t s,
                 double *rel)
{
    PCD_TRY(ws.reserve((size_t)H * ld));
    SolveArgs a{};
    a.W = W; a.H = H; a.ld = ld;
    a.stop = PCD_STOP_REL_RESIDUAL;
    PCD_CUDA(cudaMemsetAsync(ws.ctl, 0, sizeof(Ctl), s));
    const int rblocks = grid_blocks((long)W * H);
    k_mask<<<rblocks, kThreads, 0, s>>>(b, ws.mask, W, H, ld, ws.ctl);
    PCD_LAUNCHED(1);
    k_residual64<true><<<rblocks, kThreads, 0, s>>>(phi, b, ws.mask, ws.ctl, ws.partials, a, 0, 1, 0);
    PCD_LAUNCHED(1);
    PCD_CUDA(cudaMemcpyAsync(ws.ctl_host, ws.ctl, sizeof(Ctl), cudaMemcpyDeviceToHost, s));
    PCD_CUDA(cudaStreamSynchronize(s));
    *rel = ws.ctl_host[0].rel;
    return PCD_OK;
}

int enqueue_smooth(const double *b, double *phi, uint8_t *mask, Ctl *ctl, double *partials, int W, int H, int ld,
                   int sweeps, double omega, cudaStream_t s)
{
    SolveArgs a{};
    a.W = W; a.H = H; a.ld = ld;
    a.stop = PCD_STOP_REL_RESIDUAL;
    a.max_iter = sweeps;
    a.tol = 0.0;
    a.omega = omega;
    for (int c = 0; c < 5; c++) {
        a.w64[c] = omega / (double)c;
        a.w32[c] = (float)omega / (float)c;
    }
    PCD_CUDA(cudaMemsetAsync(ctl, 0, sizeof(Ctl), s));
    const int rblocks = grid_blocks((long)W * H);
    k_mask<<<rblocks, kThreads, 0, s>>>(b, mask, W, H, ld, ctl);
    PCD_LAUNCHED(1);
    const int half = (W + 1) >> 1;
    const int blocks = ceil_div((long)H * half, kThreads);
    for (int k = 0; k < sweeps; k++)
        for (int color = 0; color < 2; color++) {
            k_rb_half<double, true, false><<<blocks, kThreads, 0, s>>>(phi, b, mask, ctl, a, color, color);
            PCD_LAUNCHED(1);
        }
    k_residual64<true><<<rblocks, kThreads, 0, s>>>(phi, b, mask, ctl, partials, a, 0, 1, 0);
    PCD_LAUNCHED(1);
    return PCD_OK;
}

int enqueue_smooth_mixed(const double *b, double *phi, float *e32, float *r32, Ctl *ctl, double *partials, int W,
                         int H, int ld, int sweeps, int dev, cudaStream_t s)
{
    ClusterPlan plan{};
    if (cluster_plan(dev, W, H, 4, &plan) != PCD_OK) {
        set_error("mixed smoothing: the grid does not fit one cluster");
        return PCD_BAD_ARG;
    }
    SolveArgs a{};
    a.W = W; a.H = H; a.ld = ld;
    a.stop = PCD_STOP_REL_RESIDUAL;
    a.max_iter = sweeps;
    a.tol = 0.0;
    a.omega = 1.0;
    for (int c = 0; c < 5; c++) {
        a.w64[c] = 1.0 / (double)c;
        a.w32[c] = 1.0f / (float)c;
    }
    PCD_CUDA(cudaMemsetAsync(ctl, 0, sizeof(Ctl), s));
    PCD_CUDA(cudaMemsetAsync(e32, 0, sizeof(float) * (size_t)H * ld, s));
    const int rblocks = grid_blocks((long)W * H);
    // r32 = b - L phi and ||b|| (FP64)
    k_refine_residual<false><<<rblocks, kThreads, 0, s>>>(phi, e32, b, nullptr, r32, ctl, partials, a, 1);
    PCD_LAUNCHED(1);
    // `sweeps` FP32 Gauss-Seidel sweeps of L e = r32 on one cluster (no
    // estimates, no early end: tolerance 0, drop 0, one cycle of `sweeps`)
    ClusterArgs ca{};
    ca.W = W; ca.H = H; ca.ld = ld; ca.khp = plan.khp;
    ca.e = e32; ca.r32 = r32; ca.ctl = ctl;
    ca.check_every = sweeps + 1;
    ca.cycle_cap = sweeps;
    ca.max_iter = sweeps;
    ca.tol = 0.0;
    ca.drop = 0.0;
    for (int c = 0; c < 5; c++) ca.w32[c] = a.w32[c];
    ca.one_minus_omega = 0.0f;
    ca.depth = plan.depth;
    PCD_TRY(launch_cluster(ca, plan, s));
    // ||b - L (phi + e)|| / ||b|| in FP64 into ctl->rel, then phi += e
    k_refine_residual<false><<<rblocks, kThreads, 0, s>>>(phi, e32, b, nullptr, r32, ctl, partials, a, 0);
    PCD_LAUNCHED(1);
    k_refine_update<<<rblocks, kThreads, 0, s>>>(phi, e32, ctl, a);
    PCD_LAUNCHED(1);
    return PCD_OK;
}

bool smooth_mixed_applies(int dev, int W, int H)
{
    ClusterPlan plan{};
    return cluster_plan(dev, W, H, 4, &plan) == PCD_OK;
}

size_t residual_partials_bytes() { return sizeof(double) * 3 * kResidualBlocksMax; }

int smooth_residual(SolverWorkspace &ws, const double *b, double *phi, int W, int H, int ld, int sweeps, double omega,
                    cudaStream_t s, double *rel)
{
    PCD_TRY(ws.reserve((size_t)H * ld));
    PCD_TRY(enqueue_smooth(b, phi, ws.mask, ws.ctl, ws.partials, W, H, ld, sweeps, omega, s));
    PCD_CUDA(cudaMemcpyAsync(ws.ctl_host, ws.ctl, sizeof(Ctl), cudaMemcpyDeviceToHost, s));
    PCD_CUDA(cudaStreamSynchronize(s));
    *rel = ws.ctl_host[0].rel;
    return PCD_OK;
}

int zero_grid(double *phi, int W, int H, int ld, cudaStream_t s)
{
    k_fill<<<grid_blocks((long)W * H), kThreads, 0, s>>>(phi, W, H, ld, 0.0);
    PCD_LAUNCHED(1);
    return PCD_OK;
}

int solve_device(SolverWorkspace &ws, const double *b, double *phi, int W, int H, int ld, const pcd_solve_opts &o,
                 pcd_solve_stats *stats, cudaStream_t s)
{
    if (W < 1 || H < 1 || ld < W || !b || !phi) {
        set_error("pcd solve: bad grid arguments");
        return PCD_BAD_ARG;
    }
    if (o.max_iterations < 0 || o.stop < 0 || o.stop > 1 || o.precision < 0 || o.precision > 1) {
        set_error("pcd solve: bad options");
        return PCD_BAD_ARG;
    }
    PCD_TRY(ws.reserve((size_t)H * std::max<size_t>(ld, quads::quad_row_floats(W))));

    SolveArgs a;
    a.W = W; a.H = H; a.ld = ld;
    a.stop = o.stop;
    a.max_iter = o.max_iterations;
    a.tol = o.tol;
    a.omega = resolve_omega(o.omega, W, H);
    for (int c = 0; c < 5; c++) {
        a.w64[c] = a.omega / (double)c;             // solver.cpp:47 divides omega by cnt
        a.w32[c] = (float)a.omega / (float)c;
    }
    const int precision = o.precision;

    PCD_CUDA(cudaEventRecord(ws.t0, s));
    const int rblocks = grid_blocks((long)W * H);
    const bool mixed = precision == PCD_PREC_MIXED;
    ResidentPlan rp;
    ResidentRule rule;
    const int resident = a.max_iter > 0 ? resident_rule(ws, a, o, &rp, &rule) : PCD_BAD_ARG;
    if (resident != PCD_OK && resident != PCD_BAD_ARG) return resident;
    // mask, initial FP64 residual and norms (valid with or without NaN cells);
    // r64 for the mixed schedules that carry the residual on; r32 in the layout
    // of the schedule that will most likely run (NaN cells are not known yet)
    bool r32_quads = false;
    auto start = [&](bool in_quads) -> int {
        r32_quads = in_quads;
        PCD_CUDA(cudaMemsetAsync(ws.ctl, 0, sizeof(Ctl), s));
        return launch_start(b, phi, ws.mask, mixed && resident != PCD_OK ? ws.r64 : nullptr, mixed ? ws.r32 : nullptr,
                            ws.ctl, ws.partials, kResidualBlocksMax, a, !o.warm_start, in_quads,
                            a.stop == PCD_STOP_REL_RESIDUAL, s);
    };
    PCD_TRY(start(mixed && (resident == PCD_OK || o.schedule == PCD_SCHED_AUTO ||
                            (o.schedule == PCD_SCHED_TILES && W % 8 == 0))));
    if (resident == PCD_OK) {
        int nans = 0;
        const int st = solve_resident(ws, b, phi, a, o, rp, rule, stats, &nans, s);
        if (!nans) return st;
    }
    if (stats) stats->sweep_form = 0;  // (tile passes set their own)
    PCD_CUDA(cudaMemcpyAsync(ws.ctl_host, ws.ctl, sizeof(Ctl), cudaMemcpyDeviceToHost, s));
    PCD_CUDA(cudaStreamSynchronize(s));
    const int masked = ws.ctl_host[0].nan_cells > 0 ? 1 : 0;
    const bool done_already = ws.ctl_host[0].converged != 0 || a.max_iter == 0;

    // FP64 sweeps: the block schedule (on chip, 2-D blocks, one L2 exchange per
    // K sweeps) before the persistent bands (one per half sweep, 16.0 us a
    // 512^2 sweep) and the stripes
    const bool auto_blocks = o.schedule == PCD_SCHED_AUTO && precision == PCD_PREC_FP64 &&
                             (long)W * H >= kTileMinCells;
    if (!done_already && !masked && (o.schedule == PCD_SCHED_BLOCKS || auto_blocks)) {
        BlocksPlan bp{};
        int st = PCD_BAD_ARG;
        if (o.block_sweeps < 0 || o.block_sweeps > 8) {
            set_error("pcd solve: block_sweeps must be 0 (auto) or 1..8");
            return PCD_BAD_ARG;
        }
        st = cached_plan(ws, {kPlanBlocks, W, H, o.block_sweeps, mixed ? 1 : 0}, &bp, [&](BlocksPlan *p) {
            if (o.block_sweeps > 0) return blocks_plan(ws.dev, W, H, o.block_sweeps, mixed, p);
            int r = PCD_BAD_ARG;
            for (int K : {mixed ? 8 : 4, 4, 2, 1})
                if ((r = blocks_plan(ws.dev, W, H, K, mixed, p)) == PCD_OK) break;
            return r;
        });
        if (st == PCD_OK)
            return mixed ? solve_blocks(ws, b, phi, a, o, bp, stats, s) : solve_blocks64(ws, b, phi, a, o, bp, stats, s);
    }
    if (!done_already && !masked && precision == PCD_PREC_MIXED && a.stop == PCD_STOP_REL_RESIDUAL &&
        (o.schedule == PCD_SCHED_AUTO || o.schedule == PCD_SCHED_CLUSTER)) {
        ClusterPlan plan{};
        if (cluster_plan(ws.dev, W, H, 4, &plan) == PCD_OK) {
            if (r32_quads) PCD_TRY(start(false));
            return solve_cluster(ws, b, phi, a, o, plan, stats, s);
        }
    }
    // FP32 sweeps beyond one cluster: the tile passes before the persistent
    // schedule (measured 2-3.5x faster from 64^2 to 1024^2)
    TilePlan tp_probe;
    const bool prefer_tiles = precision == PCD_PREC_MIXED && o.schedule != PCD_SCHED_PERSISTENT &&
                              (long)W * H >= kTileMinCells && tile_grid(W, ld) &&
                              tile_plan(ws.dev, W, H, 4, &tp_probe) == PCD_OK;
    // AUTO beyond the chip's registers: widths and rows that the tile passes do not
    // take under their own name run on them, too, with the stop tests, and under
    // the name, of the schedule whose place they take: the persistent bands (chunks
    // of 32 or 16 sweeps, tested at their ends), else the stream passes (two
    // sweeps or one), else the stripes (every sweep).  1500^2: 3.2 us a sweep with
    // its refreshes, the stream passes 22.9; 9.1 and 24.5 to the max-update stop.
    TilePlan tp;
    if (!done_already && !masked && mixed && !prefer_tiles && o.schedule == PCD_SCHED_AUTO && W >= 16 && H >= 16 &&
        ld < kRefreshLdMax && (long)W * H >= kTileMinCells) {
        int G = 0, chunk = mixed_chunk(a, o), nsw = 1, name = PCD_SCHED_STRIPES;
        size_t smem = 0;
        StreamPlan probe;
        const bool bands = persist_grid(ws.dev, W, H, true, &G, &smem) == PCD_OK;
        if (bands) {
            name = PCD_SCHED_PERSISTENT;
            chunk = o.check_every > 0 ? o.check_every : (a.stop == PCD_STOP_MAX_UPDATE ? 16 : 32);
            if (o.refine_every > 0 && o.refine_every < chunk) chunk = o.refine_every;
        } else if (stream_plan(ws.dev, W, H, ld, true, &probe) == PCD_OK) {
            name = PCD_SCHED_STREAM;
            if (probe.two) nsw = 2;
        }
        if (bands || a.stop != PCD_STOP_MAX_UPDATE) nsw = 4;
        chunk = std::min(chunk, a.max_iter);
        if (tile_plan(ws.dev, W, H, nsw <= 2 ? 2 : 4, &tp) == PCD_OK) {
            if (!r32_quads) PCD_TRY(start(true));
            return solve_tiles(ws, b, phi, a, tp, nsw, chunk, !bands, name, stats, s);
        }
    }
    if (!done_already && !masked && !prefer_tiles &&
        (o.schedule == PCD_SCHED_AUTO || o.schedule == PCD_SCHED_PERSISTENT || o.schedule == PCD_SCHED_CLUSTER)) {
        int G = 0;
        size_t smem = 0;
        if (persist_grid(ws.dev, W, H, precision == PCD_PREC_MIXED, &G, &smem) == PCD_OK)
            return solve_persistent(ws, b, phi, a, precision, o, G, smem, stats, s);
    }

    if (done_already) {
        int one = 1;
        PCD_CUDA(cudaMemcpyAsync(&ws.ctl->halt, &one, sizeof(int), cudaMemcpyHostToDevice, s));
        PCD_CUDA(cudaMemcpyAsync(&ws.ctl->done, &one, sizeof(int), cudaMemcpyHostToDevice, s));
    }

    // HBM grids without NaN cells: ping-pong tile passes or stream sweeps
    // (FP32), else fused in-place stripe sweeps (grids with at least 3 rows)
    int sched = PCD_SCHED_LAUNCHES;
    StreamPlan sp;
    if (!masked && precision == PCD_PREC_MIXED && o.schedule != PCD_SCHED_STREAM &&
        o.schedule != PCD_SCHED_LAUNCHES && o.schedule != PCD_SCHED_STRIPES) {
        // register-resident tile passes; check_every: sweeps per pass (stop
        // tests after every pass), 4 at most
        const int nsw = o.check_every > 0 ? std::min(o.check_every, 4) : 4;
        if (tile_grid(W, ld) && tile_plan(ws.dev, W, H, nsw <= 2 ? 2 : 4, &tp) == PCD_OK) {
            sched = PCD_SCHED_TILES;
            if (!done_already) {
                if (!r32_quads) PCD_TRY(start(true));
                return solve_tiles(ws, b, phi, a, tp, nsw, mixed_chunk(a, o), true, PCD_SCHED_TILES, stats, s);
            }
        }
    }
    if (sched == PCD_SCHED_TILES) {
        // nothing left to sweep
    } else if (!masked && precision == PCD_PREC_MIXED &&
               (o.schedule == PCD_SCHED_AUTO || o.schedule == PCD_SCHED_STREAM ||
                o.schedule == PCD_SCHED_PERSISTENT || o.schedule == PCD_SCHED_CLUSTER ||
                o.schedule == PCD_SCHED_TILES) &&
               stream_plan(ws.dev, W, H, ld, true, &sp) == PCD_OK) {
        sched = PCD_SCHED_STREAM;
    } else if (!masked && H >= 3 && W <= 2 * kRowCellsMax * kStripeThreads && o.schedule != PCD_SCHED_LAUNCHES) {
        sched = PCD_SCHED_STRIPES;
    }
    // (r32, the first right-hand side of the FP32 sweeps, is the start's)
    if (!done_already && mixed && r32_quads) PCD_TRY(start(false));
    if (!done_already && precision == PCD_PREC_MIXED)
        PCD_CUDA(cudaMemsetAsync(ws.e32, 0, sizeof(float) * (size_t)H * ld, s));
    const bool stripes = sched == PCD_SCHED_STRIPES;
    if (stripes && ws.stripe_resident == 0) {
        int sms = 0, bps = 0;
        PCD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ws.dev));
        PCD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, k_stripe_a<double, false, 4>, kStripeThreads, 0));
        ws.stripe_resident = std::max(1, bps) * sms;
    }
    int chunk = precision == PCD_PREC_MIXED ? mixed_chunk(a, o)
                : a.stop == PCD_STOP_MAX_UPDATE ? 32 : o.check_every > 0 ? o.check_every : 32;
    if (chunk > a.max_iter && a.max_iter > 0) chunk = a.max_iter;

    SolverWorkspace::GraphEntry *ge = nullptr;
    if (!done_already) PCD_TRY(get_chunk_graph(ws, b, phi, a, precision, masked, chunk, s, &ge, sched, sp));

    PCD_CUDA(cudaEventRecord(ws.k0, s));
    // Chunk loop: launch chunk i+1 before inspecting chunk i's control block.
    const long max_chunks = a.max_iter > 0 ? (long)a.max_iter / chunk + 3 : 0;
    long launched = 0;
    int finished = done_already;
    auto flag_done = [&](const Ctl &c) { return precision == PCD_PREC_MIXED ? c.done : c.halt; };
    while (!finished) {
        if (launched >= max_chunks) {
            set_error("pcd solve: chunk budget exceeded without a halt flag");
            return PCD_TIMEOUT;
        }
        PCD_CUDA(cudaGraphLaunch(ge->exec, s));
        count_launches(ge->nodes);
        const int slot = (int)(launched & 1);
        PCD_CUDA(cudaMemcpyAsync(&ws.ctl_host[slot], ws.ctl, sizeof(Ctl), cudaMemcpyDeviceToHost, s));
        PCD_CUDA(cudaEventRecord(ws.ev[slot], s));
        launched++;
        if (launched >= 2) {
            const int prev = (int)((launched - 2) & 1);
            PCD_CUDA(cudaEventSynchronize(ws.ev[prev]));
            if (flag_done(ws.ctl_host[prev]) || ws.ctl_host[prev].error) finished = 1;
        }
    }
    PCD_CUDA(cudaEventRecord(ws.k1, s));
    // Final statistics (FP64 residual of the returned phi).
    if (precision != PCD_PREC_MIXED) {
        if (masked)
            k_residual64<true><<<rblocks, kThreads, 0, s>>>(phi, b, ws.mask, ws.ctl, ws.partials, a, 0, 1, 0);
        else
            k_residual64<false><<<rblocks, kThreads, 0, s>>>(phi, b, ws.mask, ws.ctl, ws.partials, a, 0, 1, 0);
        PCD_LAUNCHED(1);
    }
    PCD_CUDA(cudaEventRecord(ws.t1, s));
    PCD_CUDA(cudaMemcpyAsync(&ws.ctl_host[0], ws.ctl, sizeof(Ctl), cudaMemcpyDeviceToHost, s));
    PCD_CUDA(cudaStreamSynchronize(s));
    const Ctl &c = ws.ctl_host[0];
    if (c.error) {
        set_error("stream SOR: a bounded device wait gave up (status " + std::to_string(c.error) + ")");
        return c.error;
    }
    if (stats) {
        stats->sweeps = c.sweeps;
        stats->converged = c.converged;
        stats->rel_residual = c.rel;
        stats->max_residual = c.rmax;
        stats->last_max_update = c.last_max;
        stats->residual_checks = c.checks;
        float ms = 0.f;
        cudaEventElapsedTime(&ms, ws.t0, ws.t1);
        stats->device_ms = ms;
        cudaEventElapsedTime(&ms, ws.k0, ws.k1);
        stats->sweep_ms = ms;
        stats->schedule_used = sched;
    }
    return c.converged ? PCD_OK : PCD_NOT_CONVERGED;
}


// ---------------------------------------------------------------------------
// Batched tile solve: the grids of a batch share one tile pass per launch
// (k_tile_batch) and one FP64 refresh per chunk of passes, each
// grid with its own control block, so a grid that has converged drops out
// while the others go on.
namespace {

// Most blocks of one grid in the batched FP64 refresh.
constexpr int kBatchRefineBlocks = 1024;

}  // namespace

int TileBatchWorkspace::reserve(size_t cells, int count, int tiles)
{
    // per cell: the two corrections, the right-hand side, the second potential
    if (cells > arena_cells) {
        for (auto &kv : graphs) cudaGraphExecDestroy(kv.second);
        graphs.clear();
        if (arena) cudaFree(arena);
        if (phi2) cudaFree(phi2);
        arena = nullptr;
        phi2 = nullptr;
        arena_cells = 0;
        PCD_CUDA(cudaMalloc(&arena, 3 * cells * sizeof(float)));
        PCD_CUDA(cudaMalloc(&phi2, cells * sizeof(double)));
        arena_cells = cells;
    }
    if (count > cap) {
        for (auto &kv : graphs) cudaGraphExecDestroy(kv.second);
        graphs.clear();
        if (ctl) cudaFree(ctl);
        if (ctl_host) cudaFreeHost(ctl_host);
        if (partials) cudaFree(partials);
        if (jobs) cudaFree(jobs);
        if (rjobs) cudaFree(rjobs);
        ctl = nullptr; ctl_host = nullptr; partials = nullptr; jobs = nullptr; rjobs = nullptr;
        cap = 0;
        PCD_CUDA(cudaMalloc(&ctl, sizeof(Ctl) * count));
        PCD_CUDA(cudaMallocHost(&ctl_host, 2 * sizeof(Ctl) * count));
        PCD_CUDA(cudaMalloc(&partials, sizeof(double) * 3 * kBatchRefineBlocks * count));
        PCD_CUDA(cudaMalloc(&jobs, sizeof(TileJob) * count));
        PCD_CUDA(cudaMalloc(&rjobs, sizeof(RefreshJob) * count));
        cap = count;
    }
    if (!t0) {
        PCD_CUDA(cudaEventCreate(&t0));
        PCD_CUDA(cudaEventCreate(&t1));
        PCD_CUDA(cudaEventCreateWithFlags(&ev[0], cudaEventDisableTiming));
        PCD_CUDA(cudaEventCreateWithFlags(&ev[1], cudaEventDisableTiming));
    }
    if (tiles > sync_tiles) {
        for (auto &kv : graphs) cudaGraphExecDestroy(kv.second);
        graphs.clear();
        if (sync) cudaFree(sync);
        sync = nullptr;
        sync_tiles = 0;
        PCD_CUDA(cudaMalloc(&sync, sizeof(unsigned) * (2 + (size_t)tiles)));
        sync_tiles = tiles;
    }
    return PCD_OK;
}

void TileBatchWorkspace::release()
{
    for (auto &kv : graphs) cudaGraphExecDestroy(kv.second);
    graphs.clear();
    if (arena) cudaFree(arena);
    if (phi2) cudaFree(phi2);
    if (ctl) cudaFree(ctl);
    if (ctl_host) cudaFreeHost(ctl_host);
    if (partials) cudaFree(partials);
    if (jobs) cudaFree(jobs);
    if (rjobs) cudaFree(rjobs);
    if (sync) cudaFree(sync);
    for (cudaEvent_t *e : {&t0, &t1, &ev[0], &ev[1]})
        if (*e) cudaEventDestroy(*e);
    *this = TileBatchWorkspace();
}

bool batch_tiles_apply(const pcd_instance *inst, int count)
{
    if (!inst || count < 1 || count > kTileBatchJobsMax) return false;
    for (int i = 0; i < count; i++) {
        const pcd_instance &q = inst[i];
        if (!q.b || !q.phi || q.width < 8 || q.height < 1 || q.width % 8 != 0 || q.ld < q.width || q.ld % 4 != 0 ||
            q.ld >= kRefreshLdMax)
            return false;
    }
    return true;
}

int batch_tiles_solve(TileBatchWorkspace &ws, int dev, const pcd_instance *inst, int count, const pcd_solve_opts &o,
                      pcd_instance_stats *stats, pcd_batch_stats *bstats, cudaStream_t s)
{
    if (!batch_tiles_apply(inst, count)) {
        set_error("batched tile solve: every grid needs a width that is a multiple of 8 and ld a multiple of 4, "
                  "and at most " + std::to_string(kTileBatchJobsMax) + " grids");
        return PCD_BAD_ARG;
    }
    if (o.stop != PCD_STOP_REL_RESIDUAL || !(o.tol > 0.0) || o.max_iterations < 1) {
        set_error("pcd_batch_solve_device: the batch solve takes the relative-residual stop with tol > 0");
        return PCD_BAD_ARG;
    }
    size_t smem = 0;
    int grid = 0, sms = 0;
    PCD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    bool narrow = false;
    for (int i = 0; i < count; i++) narrow = narrow || inst[i].width == 8;
    PCD_TRY(tile_batch_config(dev, count, narrow, &smem, &grid));
    size_t per = 0;
    for (int i = 0; i < count; i++) per += (size_t)inst[i].height * inst[i].ld;
    PCD_TRY(ws.reserve(per, count, 0));

    // largest grids first: their refresh blocks are dispatched first
    std::vector<int> order(count);
    for (int i = 0; i < count; i++) order[i] = i;
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) {
        return (long)inst[x].width * inst[x].height > (long)inst[y].width * inst[y].height;
    });
    std::vector<TileJob> tj((size_t)count);
    std::vector<RefreshJob> rj((size_t)count);
    size_t off = 0, all_cells = 0;
    for (int i = 0; i < count; i++) all_cells += (size_t)inst[i].width * inst[i].height;
    int tiles = 0, blocks = 0, maxdim = 0;
    for (int k = 0; k < count; k++) {
        const int i = order[k];
        const pcd_instance &q = inst[i];
        maxdim = std::max(maxdim, std::max(q.width, q.height));
        TileJob &t = tj[k];
        RefreshJob &r = rj[k];
        t.ea = ws.arena + off;
        t.eb = ws.arena + per + off;
        t.r32 = ws.arena + 2 * per + off;
        t.ctl = ws.ctl + k;
        t.W = q.width;
        t.H = q.height;
        PCD_TRY(tile_job_setup(&t));
        t.tile0 = tiles;
        t.max_iter = o.max_iterations;
        const double om = resolve_omega(o.omega, q.width, q.height);
        for (int c = 0; c < 5; c++) t.w32[c] = (float)om / (float)c;
        tiles += t.ncol * t.nrow;
        r.b = q.b;
        r.phi = q.phi;
        r.phi2 = ws.phi2 + off;
        r.e0 = t.ea;
        r.e1 = t.eb;
        r.r32 = ws.arena + 2 * per + off;
        r.ctl = t.ctl;
        r.error = &ws.ctl->error;
        r.partials = ws.partials + (size_t)3 * kBatchRefineBlocks * k;
        r.W = q.width;
        r.H = q.height;
        r.ld = q.ld;
        r.blk0 = blocks;
        r.nblk = refresh_shape(q.width, q.height, q.ld, kBatchRefineBlocks,
                               sms * ((double)q.width * q.height / (double)all_cells), &r.rows);
        blocks += r.nblk;
        off += (size_t)q.height * q.ld;
    }
    PCD_TRY(ws.reserve(per, count, tiles));
    const TileJob *d_jobs = static_cast<const TileJob *>(ws.jobs);
    const RefreshJob *d_rjobs = static_cast<const RefreshJob *>(ws.rjobs);
    // sweeps between FP64 refreshes (passes of 4, the last one shorter):
    // refine_every, else 128 when the largest side is 1024 or more, down to
    // 32 when it is 256 or less
    const int spacing = o.refine_every > 0 ? o.refine_every : 4 * std::max(8, std::min(32, maxdim / 32));
    const int chunk = std::min({spacing, o.max_iterations, kChunkSweepsMax});

    PCD_CUDA(cudaEventRecord(ws.t0, s));
    PCD_CUDA(cudaMemcpyAsync(ws.jobs, tj.data(), sizeof(TileJob) * count, cudaMemcpyHostToDevice, s));
    PCD_CUDA(cudaMemcpyAsync(ws.rjobs, rj.data(), sizeof(RefreshJob) * count, cudaMemcpyHostToDevice, s));
    PCD_CUDA(cudaMemsetAsync(ws.ctl, 0, sizeof(Ctl) * count, s));
    PCD_CUDA(cudaMemsetAsync(ws.sync, 0, sizeof(unsigned) * (2 + (size_t)tiles), s));
    // first right-hand side, ||b|| and the stop test of the starting phi
    PCD_TRY(launch_first_refresh(d_rjobs, count, blocks, o.tol, !o.warm_start, s));

    // one CUDA graph per batch signature: the chunk's sweeps and the refresh
    const long long limit = ws.wait_limit > 0 ? ws.wait_limit : kWordPolls;
    std::vector<long long> key = {count, tiles, blocks, chunk, narrow, grid, (long long)smem, limit, ws.withhold_flag,
                                  (long long)(uintptr_t)ws.jobs, (long long)(uintptr_t)ws.rjobs,
                                  (long long)(uintptr_t)ws.sync};
    {
        long long tb;
        std::memcpy(&tb, &o.tol, 8);
        key.push_back(tb);
    }
    cudaGraphExec_t exec = nullptr;
    auto it = ws.graphs.find(key);
    if (it != ws.graphs.end()) {
        exec = it->second;
    } else {
        cudaGraph_t g;
        PCD_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
        int st = launch_tile_batch(d_jobs, count, tiles, chunk, narrow, grid, smem, ws.sync, ws.sync + 2, limit,
                                   ws.withhold_flag, s);
        if (st == PCD_OK) st = launch_refresh(d_rjobs, RefreshJob{}, count, blocks, o.tol, s);
        cudaError_t ce = cudaStreamEndCapture(s, &g);
        if (st != PCD_OK) {
            if (ce == cudaSuccess) cudaGraphDestroy(g);
            return st;
        }
        if (ce != cudaSuccess) {
            set_error(std::string("batched tile graph capture: ") + cudaGetErrorString(ce));
            return PCD_DEVICE_ERROR;
        }
        ce = cudaGraphInstantiate(&exec, g, 0);
        cudaGraphDestroy(g);
        if (ce != cudaSuccess) {
            set_error(std::string("batched tile graph instantiate: ") + cudaGetErrorString(ce));
            return PCD_DEVICE_ERROR;
        }
        if (ws.graphs.size() > 16) {
            for (auto &kv : ws.graphs) cudaGraphExecDestroy(kv.second);
            ws.graphs.clear();
        }
        ws.graphs[key] = exec;
    }

    // chunk i+1 is launched before chunk i's control blocks are inspected
    const long max_chunks = (long)o.max_iterations / chunk + 3;
    long launched = 0;
    bool finished = false;
    auto all_done = [&](const Ctl *c) {
        if (c[0].error) return true;  // (the batch's)
        for (int i = 0; i < count; i++)
            if (!c[i].done) return false;
        return true;
    };
    while (!finished) {
        if (launched >= max_chunks) {
            set_error("batched tile solve: chunk budget exceeded without every grid done");
            return PCD_TIMEOUT;
        }
        PCD_CUDA(cudaGraphLaunch(exec, s));
        count_launches(2);
        const int slot = (int)(launched & 1);
        PCD_CUDA(cudaMemcpyAsync(ws.ctl_host + (size_t)slot * count, ws.ctl, sizeof(Ctl) * count,
                                 cudaMemcpyDeviceToHost, s));
        PCD_CUDA(cudaEventRecord(ws.ev[slot], s));
        launched++;
        if (launched >= 2) {
            const int prev = (int)((launched - 2) & 1);
            PCD_CUDA(cudaEventSynchronize(ws.ev[prev]));
            if (all_done(ws.ctl_host + (size_t)prev * count)) finished = true;
        }
    }
    PCD_TRY(launch_phi_settle(d_rjobs, count, s));
    PCD_CUDA(cudaEventRecord(ws.t1, s));
    PCD_CUDA(cudaMemcpyAsync(ws.ctl_host, ws.ctl, sizeof(Ctl) * count, cudaMemcpyDeviceToHost, s));
    PCD_CUDA(cudaStreamSynchronize(s));
    if (ws.ctl_host[0].error) {
        set_error("batched tile solve: a bounded device wait gave up");
        return ws.ctl_host[0].error;
    }
    float ms = 0.f;
    cudaEventElapsedTime(&ms, ws.t0, ws.t1);
    int all = 1;
    long long cell_sweeps = 0;
    for (int k = 0; k < count; k++) {
        const int i = order[k];
        const Ctl &c = ws.ctl_host[k];
        if (stats) {
            stats[i].sweeps = c.sweeps;
            stats[i].converged = c.converged;
            stats[i].rel_residual = c.rel;
            stats[i].cycles = c.checks;
        }
        all &= c.converged;
        cell_sweeps += (long long)inst[i].width * inst[i].height * c.sweeps;
    }
    if (bstats) {
        bstats->device_ms = ms;
        bstats->clusters = 0;
        bstats->cluster_size = 0;
        bstats->smem_bytes = (long long)smem;
        bstats->cell_sweeps = cell_sweeps;
        bstats->check_every = spacing;
        bstats->refine_drop = 0.0;
        bstats->tuned = 0;
    }
    return all ? PCD_OK : PCD_NOT_CONVERGED;
}

}  // namespace pcd
