// refresh.cu -- the FP64 passes of a solve (sm_103a).
//
// This part runs an FP64 operation of a warp every 16 clocks of an SM (1/56 of
// the FP32 rate), so these passes are bound by the number of FP64 instructions,
// not by memory: 20 bytes read and 12 written a cell take 80 us at 4096^2, six
// FP64 operations a cell 190.
//
// k_refresh folds the FP32 correction into the potential and renews the
// residual in one pass:  xi = phi + e,  r = b - (sum of neighbours - cnt xi).
// A warp walks down a strip of 30 columns (lanes 1 to 30; lanes 0 and 31 the
// columns beside it).  With D(x, y) = xi(x+1, y) + xi(x, y+1) the neighbour sum
// of (x, y) is D(x-1, y-1) + D(x, y), so a cell costs two additions for it
// instead of three, one shuffle each way, and xi is formed once:  add, D, D + D,
// multiply-add, subtract, multiply-add for the norm (the conversions run beside
// them).  4096^2: 308 us, 2048^2: 88, the pipe 81% busy; 386 and 122 when the
// compiler formed the neighbour counts in FP64 for every row, the largest |r| was
// compared as 64-bit words and pieces of 8, 16 or 32 rows left SMs idle at the
// end.  (One thread a cell forming xi of all five cells took about 24
// operations.)  Cells outside the grid read 0.
//
// xi goes to the other of two buffers, because a neighbouring strip may still
// need the old phi; the control block says which one holds the potential.
#include <algorithm>
#include <cmath>

#include "refresh.cuh"
#include "sor_quads.cuh"

namespace pcd {

namespace {

constexpr int kRefreshWarps = 4;      // warps of a block
constexpr int kRefreshResident = 4;   // blocks of an SM (4096^2: 305 us, with eight 330)
constexpr int kRefreshCols = 30;      // columns a warp owns
constexpr int kStartThreads = 256;

__device__ __forceinline__ int rf_load(const int *p) { return *(const volatile int *)p; }

__device__ __forceinline__ bool is_nan_bits(double v)
{
    return ((unsigned long long)__double_as_longlong(v) << 1) > 0xffe0000000000000ull;
}

// Running max of |r| on its words (they order like the values; NaN does not raise
// it), off the FP64 pipe.
__device__ __forceinline__ void max_abs_words(unsigned &mhi, unsigned &mlo, double r)
{
    const unsigned hi = (unsigned)__double2hiint(r) & 0x7fffffffu, lo = (unsigned)__double2loint(r);
    const bool more = hi > mhi || (hi == mhi && lo > mlo), number = hi < 0x7ff00000u || (hi == 0x7ff00000u && lo == 0u);
    mhi = more && number ? hi : mhi;
    mlo = more && number ? lo : mlo;
}

__device__ __forceinline__ bool rf_last_block(Ctl *ctl, int nblk)
{
    __shared__ bool is_last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        is_last = atomicAdd(&ctl->blocks_done_r, 1u) == (unsigned)nblk - 1u;
    }
    __syncthreads();
    if (is_last) __threadfence();
    return is_last;
}

// The control block into host memory, one thread (the end of the launch, which
// the host waits for, makes it visible).
__device__ void rf_report(const Ctl *ctl, Ctl *report)
{
    static_assert(sizeof(Ctl) % 8 == 0, "copied in 64-bit words");
    const volatile unsigned long long *from = reinterpret_cast<const volatile unsigned long long *>(ctl);
    volatile unsigned long long *to = reinterpret_cast<volatile unsigned long long *>(report);
#pragma unroll
    for (int k = 0; k < (int)(sizeof(Ctl) / 8); k++) to[k] = from[k];
}

// The norms of a pass: sums of r^2 and b^2 and the largest |r|'s words.
struct Norms {
    double rr = 0.0, bb = 0.0;
    unsigned hi = 0u, lo = 0u;
    __device__ __forceinline__ double rmax() const { return __hiloint2double((int)hi, (int)lo); }
};

// The block's norms in thread 0, in a fixed order (every thread calls).  FP64
// instructions are what it would wait for: five a sum and warp, none for the
// maximum, and no sum that is not asked for.  (Three FP64 reductions, and
// partials loaded one after the other: 23 us a 512^2 refresh, now 17.)
template <bool BB>
__device__ __forceinline__ void rf_block_norms(Norms &v)
{
    __shared__ Norms part[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (int)(blockDim.x >> 5);
    v.rr = warp_sum(v.rr);
    if (BB) v.bb = warp_sum(v.bb);
    const unsigned hi = __reduce_max_sync(0xffffffffu, v.hi);
    v.lo = __reduce_max_sync(0xffffffffu, v.hi == hi ? v.lo : 0u);
    v.hi = hi;
    __syncthreads();
    if (lane == 0) part[w] = v;
    __syncthreads();
    if (threadIdx.x != 0) return;
    for (int k = 1; k < nw; k++) {
        const Norms &p = part[k];
        v.rr += p.rr;
        if (BB) v.bb += p.bb;
        if (p.hi > v.hi || (p.hi == v.hi && p.lo > v.lo)) {
            v.hi = p.hi;
            v.lo = p.lo;
        }
    }
}

// The blocks' norms (three doubles each) in thread 0 of the last block, in a fixed
// order.
template <bool BB>
__device__ __forceinline__ Norms rf_all_norms(const double *partials, int nblk)
{
    Norms v;
    for (int k0 = threadIdx.x; k0 < nblk; k0 += 4 * blockDim.x) {
        double r[4], b[4], m[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int k = k0 + u * (int)blockDim.x;
            const bool in = k < nblk;
            r[u] = in ? __ldcg(partials + 3 * k) : 0.0;
            b[u] = BB && in ? __ldcg(partials + 3 * k + 1) : 0.0;
            m[u] = in ? __ldcg(partials + 3 * k + 2) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            v.rr += r[u];
            if (BB) v.bb += b[u];
            max_abs_words(v.hi, v.lo, m[u]);
        }
    }
    rf_block_norms<BB>(v);
    return v;
}

// FIRST: the start of a batch's solves (e = 0; zero: phi = 0 too, and written).
template <bool FIRST>
__global__ void __launch_bounds__(32 * kRefreshWarps)
    k_refresh(const RefreshJob *__restrict__ jobs, RefreshJob one, int njobs, double tol, int zero)
{
    RefreshJob J = one;
    if (jobs) {
        int lo = 0, hi = njobs - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (__ldg(&jobs[mid].blk0) <= (int)blockIdx.x) lo = mid;
            else hi = mid - 1;
        }
        J = jobs[lo];
    }
    Ctl *ctl = J.ctl;
    const int side = rf_load(&ctl->phi_side);
    if (rf_load(&ctl->done) | rf_load(J.error) | rf_load(&ctl->nan_cells)) {  // (loads side by side)
        if (!J.report) return;
        if ((int)blockIdx.x == J.blk0 && threadIdx.x == 0) rf_report(ctl, J.report);
        if (side)
            for (int y = (int)blockIdx.x - J.blk0; y < J.H; y += J.nblk)
                for (int x = threadIdx.x; x < J.W; x += blockDim.x)
                    J.phi[(size_t)y * J.ld + x] = J.phi2[(size_t)y * J.ld + x];
        return;
    }
    const double *__restrict__ pin = side ? J.phi2 : J.phi;
    double *__restrict__ pout = FIRST || side ? J.phi : J.phi2;
    const float *__restrict__ e = rf_load(&ctl->stream_out) ? J.e1 : J.e0;
    const int W = J.W, H = J.H, ld = J.ld, KQ = (W + 7) >> 3;
    const int lane = threadIdx.x & 31, w = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0);
    const int strips = (W + kRefreshCols - 1) / kRefreshCols, pieces = (H + J.rows - 1) / J.rows;
    Norms v;
    for (int item = ((int)blockIdx.x - J.blk0) * kRefreshWarps + w; item < strips * pieces;
         item += J.nblk * kRefreshWarps) {
        const int piece = item / strips, strip = item - piece * strips;
        const int x = strip * kRefreshCols + lane - 1;
        const bool in = x >= 0 && x < W, own = in && lane >= 1 && lane <= kRefreshCols;
        const int y0 = piece * J.rows, y1 = min(y0 + J.rows, H), yb = max(y0 - 1, 0);
        // neighbours of a cell with both vertical ones, with one and with none,
        // as the high words of doubles
        const int nh = (x > 0) + (x < W - 1);
        const int c2 = nh == 2 ? 0x40100000 : nh ? 0x40080000 : 0x40000000;
        const int c1 = nh == 2 ? 0x40080000 : nh ? 0x40000000 : 0x3ff00000;
        const int c0 = nh == 2 ? 0x40000000 : nh ? 0x3ff00000 : 0;
        // places as byte offsets in 32 bits from the piece's first row (28% fewer
        // instructions than 64-bit indices)
        const unsigned at = in ? (unsigned)x : 0u, row = (unsigned)ld * 8u, row32 = 32u * (unsigned)KQ;
        const unsigned col = (unsigned)quads::quad_column((int)at, KQ) * 4u;
        const size_t base = (size_t)yb * ld, base32 = (size_t)yb * 8 * KQ;
        const char *p_in = reinterpret_cast<const char *>(pin + base), *p_b = reinterpret_cast<const char *>(J.b + base);
        const char *p_e = reinterpret_cast<const char *>(e + base32);
        char *p_out = reinterpret_cast<char *>(pout + base), *p_r = reinterpret_cast<char *>(J.r32 + base32);
        auto load = [&](int y, double &p, float &ev) {
            const bool ok = in && y >= 0 && y < H;
            const unsigned k = (unsigned)(y - yb);
            p = 0.0;
            ev = 0.f;
            if (ok && !(FIRST && zero)) p = *reinterpret_cast<const double *>(p_in + (k * row + at * 8u));
            if (ok && !FIRST) ev = *reinterpret_cast<const float *>(p_e + (k * row32 + col));
        };
        auto load_b = [&](int y) {
            return *reinterpret_cast<const double *>(p_b + ((unsigned)(y - yb) * row + at * 8u));
        };
        // rows y0 - 1, y0 and y0 + 1; then one row ahead of the one in hand
        double pa, pb, pc, bc;
        float ea, eb, ec;
        load(y0 - 1, pa, ea);
        load(y0, pb, eb);
        load(y0 + 1, pc, ec);
        bc = own ? load_b(y0) : 0.0;
        const double xa = pa + (double)ea;
        double xc = pb + (double)eb;
        // D(x, y0 - 1)
        double dp = __shfl_down_sync(0xffffffffu, xa, 1) + xc;
        for (int y = y0; y < y1; y++) {
            double pn, bn = 0.0;
            float en;
            load(y + 2, pn, en);
            if (own && y + 1 < y1) bn = load_b(y + 1);
            const double xn = pc + (double)ec;
            const double d = __shfl_down_sync(0xffffffffu, xc, 1) + xn;
            const double sum = __shfl_up_sync(0xffffffffu, dp, 1) + d;
            const bool top = y > 0, bot = y < H - 1;
            const double cnt = __hiloint2double(top && bot ? c2 : top || bot ? c1 : c0, 0);
            const double r = fma(cnt, xc, bc) - sum;
            if (own) {
                const unsigned k = (unsigned)(y - yb);
                if (!FIRST || zero) *reinterpret_cast<double *>(p_out + (k * row + at * 8u)) = xc;
                *reinterpret_cast<float *>(p_r + (k * row32 + col)) = -(float)r;
                // (a start's norms leave out cells whose b is NaN; after a sweep their
                // correction is NaN, too, and no norm is a number any more)
                if (!FIRST || !is_nan_bits(bc)) {
                    v.rr = fma(r, r, v.rr);
                    if (FIRST) v.bb = fma(bc, bc, v.bb);
                    max_abs_words(v.hi, v.lo, r);
                }
            }
            dp = d;
            xc = xn;
            pc = pn;
            ec = en;
            bc = bn;
        }
    }
    rf_block_norms<FIRST>(v);
    if (threadIdx.x == 0) {
        double *p = J.partials + 3 * ((int)blockIdx.x - J.blk0);
        p[0] = v.rr;
        p[1] = v.bb;
        p[2] = v.rmax();
    }
    if (!rf_last_block(ctl, J.nblk)) return;
    const double bnorm = FIRST ? 0.0 : *(const volatile double *)&ctl->bnorm;
    v = rf_all_norms<FIRST>(J.partials, J.nblk);
    if (threadIdx.x == 0) {
        volatile Ctl *c = ctl;
        const double rn = sqrt(v.rr), bn = FIRST ? sqrt(v.bb) : bnorm, rel = bn > 0.0 ? rn / bn : rn;
        if (FIRST) c->bnorm = bn;
        c->rnorm = rn;
        c->rmax = v.rmax();
        c->rel = rel;
        c->checks = c->checks + 1;
        if (tol >= 0.0 && rel <= tol) {
            c->converged = 1;
            c->halt = 1;
        }
        if (c->halt) c->done = 1;
        if (!FIRST) c->phi_side = side ^ 1;
        c->stream_out = 0;
        c->blocks_done_r = 0;
        __threadfence();
        if (J.report) rf_report(ctl, J.report);
    }
}

__global__ void __launch_bounds__(kStartThreads) k_phi_settle(const RefreshJob *__restrict__ jobs)
{
    const RefreshJob &J = jobs[blockIdx.z];
    if (!rf_load(&J.ctl->phi_side)) return;
    for (int x = blockIdx.x * blockDim.x + threadIdx.x; x < J.W; x += gridDim.x * blockDim.x)
        for (int y = blockIdx.y; y < J.H; y += gridDim.y) J.phi[(size_t)y * J.ld + x] = J.phi2[(size_t)y * J.ld + x];
}

template <bool ZERO>
__global__ void __launch_bounds__(kStartThreads)
    k_start(const double *__restrict__ b, double *__restrict__ phi, uint8_t *__restrict__ mask,
            double *__restrict__ r64, float *__restrict__ r32, Ctl *ctl, double *partials, SolveArgs a, int in_quads,
            int test)
{
    const int W = a.W, H = a.H, ld = a.ld;
    Norms v;
    int nans = 0;
    const int KQ = (W + 7) >> 3;
    const int last = in_quads ? 8 * KQ : W;
    for (int x = blockIdx.x * blockDim.x + threadIdx.x; x < last; x += gridDim.x * blockDim.x) {
        const int col = quads::quad_column(x, KQ);
        for (int y = blockIdx.y; y < H; y += gridDim.y) {
            if (x >= W) {  // the rest of the last quads
                r32[(long)y * 8 * KQ + col] = 0.f;
                continue;
            }
            const size_t i = (size_t)y * ld + x;
            const bool l = x > 0 && !is_nan_bits(b[i - 1]), u = y > 0 && !is_nan_bits(b[i - ld]);
            const bool rt = x < W - 1 && !is_nan_bits(b[i + 1]), d = y < H - 1 && !is_nan_bits(b[i + ld]);
            const double bi = b[i];
            const bool nan = is_nan_bits(bi);
            mask[i] = (uint8_t)((l ? 1 : 0) | (u ? 2 : 0) | (rt ? 4 : 0) | (d ? 8 : 0) | (nan ? 16 : 0));
            double r = bi;
            if (ZERO) {
                phi[i] = 0.0;
            } else if (!nan) {
                double sum = 0.0;
                if (l) sum += phi[i - 1];
                if (u) sum += phi[i - ld];
                if (rt) sum += phi[i + 1];
                if (d) sum += phi[i + ld];
                r = bi - (sum - (double)((int)l + (int)u + (int)rt + (int)d) * phi[i]);
            }
            if (r64 && !nan) r64[i] = r;
            if (r32) {
                if (in_quads) r32[(long)y * 8 * KQ + col] = -(float)r;
                else r32[i] = (float)r;
            }
            if (nan) {
                nans++;
                continue;
            }
            if (!ZERO) v.rr = fma(r, r, v.rr);
            v.bb = fma(bi, bi, v.bb);
            max_abs_words(v.hi, v.lo, r);
        }
    }
    if (ZERO) v.rr = v.bb;
    if (nans) atomicAdd(&ctl->nan_cells, nans);
    rf_block_norms<true>(v);
    const int blk = blockIdx.y * gridDim.x + blockIdx.x, nblk = gridDim.x * gridDim.y;
    if (threadIdx.x == 0) {
        partials[3 * blk] = v.rr;
        partials[3 * blk + 1] = v.bb;
        partials[3 * blk + 2] = v.rmax();
    }
    if (!rf_last_block(ctl, nblk)) return;
    v = rf_all_norms<true>(partials, nblk);
    if (threadIdx.x == 0) {
        volatile Ctl *c = ctl;
        const double rn = sqrt(v.rr), bn = sqrt(v.bb), rel = bn > 0.0 ? rn / bn : rn;
        c->rnorm = rn;
        c->bnorm = bn;
        c->rmax = v.rmax();
        c->rel = rel;
        c->checks = c->checks + 1;
        if (test && rel <= a.tol) {
            c->converged = 1;
            c->halt = 1;
            c->done = 1;
        }
        c->blocks_done_r = 0;
        __threadfence();
    }
}

}  // namespace

int refresh_shape(int W, int H, int ld, int cap, double chip_sms, int *rows)
{
    // An SM's time is that of its warps' FP64 instructions, six a row and five
    // for the rows of overlap, on one pipe; with fewer than twelve warps on it,
    // their latency.  All blocks are resident at once, so the fullest SM counts.
    const int strips = ceil_div(W, kRefreshCols);
    const double sms = std::max(1.0, chip_sms);
    // (a piece's places are byte offsets in 32 bits: four rows more than it has)
    const int most = (int)std::max<long>(1, std::min<long>(H, (1l << 32) / (8l * ld) - 4));
    double best = 0.0;
    int best_rows = 0, best_blocks = 1;
    for (int r = std::min(4, most); r <= most; r += r < 32 ? 1 : r / 16) {
        const long blocks = ((long)strips * ceil_div(H, r) + kRefreshWarps - 1) / kRefreshWarps;
        if (blocks > kRefreshResident * sms || blocks > cap) continue;
        const double t = std::max(12.0, kRefreshWarps * std::ceil(blocks / sms)) * (6 * r + 5);
        if (best_rows && t >= best) continue;
        best = t;
        best_rows = r;
        best_blocks = (int)blocks;
    }
    if (!best_rows) {  // more pieces than warps
        best_rows = most;
        best_blocks = std::max(1, std::min<int>(cap, (int)(kRefreshResident * sms)));
    }
    *rows = best_rows;
    return best_blocks;
}

int launch_refresh(const RefreshJob *jobs, const RefreshJob &one, int njobs, int blocks, double tol, cudaStream_t s)
{
    k_refresh<false><<<blocks, 32 * kRefreshWarps, 0, s>>>(jobs, one, njobs, tol, 0);
    PCD_LAUNCHED(1);
    return PCD_OK;
}

int launch_first_refresh(const RefreshJob *jobs, int njobs, int blocks, double tol, bool zero, cudaStream_t s)
{
    k_refresh<true><<<blocks, 32 * kRefreshWarps, 0, s>>>(jobs, RefreshJob{}, njobs, tol, zero ? 1 : 0);
    PCD_LAUNCHED(1);
    return PCD_OK;
}

int launch_phi_settle(const RefreshJob *jobs, int njobs, cudaStream_t s)
{
    k_phi_settle<<<dim3(4, 64, njobs), kStartThreads, 0, s>>>(jobs);
    PCD_LAUNCHED(1);
    return PCD_OK;
}

int launch_start(const double *b, double *phi, uint8_t *mask, double *r64, float *r32, Ctl *ctl, double *partials,
                 int max_partials, const SolveArgs &a, bool zero, bool quads, bool test, cudaStream_t s)
{
    const int gx = std::min(ceil_div(quads ? quads::quad_row_floats(a.W) : a.W, kStartThreads), max_partials);
    const dim3 grid(gx, std::max(1, std::min(a.H, max_partials / gx)));
    if (zero) k_start<true><<<grid, kStartThreads, 0, s>>>(b, phi, mask, r64, r32, ctl, partials, a, quads ? 1 : 0,
                                                      test ? 1 : 0);
    else k_start<false><<<grid, kStartThreads, 0, s>>>(b, phi, mask, r64, r32, ctl, partials, a, quads ? 1 : 0,
                                                      test ? 1 : 0);
    PCD_LAUNCHED(1);
    return PCD_OK;
}

}  // namespace pcd
