// sor_blocks64.cu -- persistent FP64 red-black SOR over 2-D blocks (sm_103a):
// one cooperative launch per solve, the whole chip on one grid.
//
// The grid is cut into TY x TX blocks, one CTA each.  A CTA keeps its block
// plus a halo of h = 2K cells on every side in shared memory and runs K
// red-black sweeps between exchanges (the dependency cone of K sweeps ends
// inside the halo).  Halo cells travel as tagged words (words.cuh),
// double-buffered by epoch parity: a CTA overwrites epoch n with n + 2 only
// after it read its neighbours' n + 1, which they publish after reading n.
//
// Region: 64 columns, lane k holding the column pair (ox + 2k, ox + 2k + 1), ox
// even; plane c row r index k is the cell of colour c (colour = (x + y) & 1) of
// lane k's pair, at column ox + 2k + q with q = (c + y) & 1.  Cells outside the
// grid hold 0 and are never relaxed.
//
// Update, with w = omega / cnt:  phi' = (1 - omega) phi + w sum - w b
// (solver.cpp:47 with w cnt = omega), w b kept per cell.
//
// Bound: the FP64 pipe (a warp instruction takes 64 cycles of a scheduler).
// So a warp walks down consecutive rows with D(x, y) = phi(x+1, y) +
// phi(x, y+1): the neighbour sum of (x, y) is D(x-1, y-1) + D(x, y), four FP64
// operations a cell instead of five (and one more for a walk's first row); 8
// warps, because two of them keep a scheduler's FP64 pipe busy and longer
// walks have fewer first rows; max |delta| and |r| are compared as integers.
// Measured (us a sweep, before: five operations, flags and fences, rows dealt
// out one by one): 512^2 6.5 -> 4.36 (pipe 59% busy), 256^2 3.7 -> 2.37, 1024^2
// 17.2 -> 12.0 (72%), 64^2 1.8.  12 and 16 warps, and deeper unrolling, measured
// within 3% of this either way.
#include <algorithm>

#include "sor_blocks64.cuh"
#include "words.cuh"

namespace pcd {

namespace {

using namespace words;

constexpr int kB64Threads = 256, kB64Warps = kB64Threads / 32;
constexpr int kB64Pairs = 32;  // column pairs of a region

struct Block64 {
    int y0, y1, x0, x1, oy, ox, R, RT, h, k, warp, H;
    bool act0, act1, own0, own1;
    int cx0, cx1;                  // horizontal neighbours of the lane's two cells
    double wi0, wi1, we0, we1;     // omega / cnt in rows with two and one vertical neighbours
    double *X, *WB;                // planes: state, w b
    int ps;                        // elements of one colour's plane

    __device__ __forceinline__ double *xrow(int c, int r) const { return X + c * ps + (r + 1) * 32 + k; }
    __device__ __forceinline__ double *wbrow(int c, int r) const { return WB + c * ps + (r + 1) * 32 + k; }
    __device__ __forceinline__ double weight(int q, int cy) const
    {
        return q ? (cy == 2 ? wi1 : we1) : (cy == 2 ? wi0 : we0);
    }
    __device__ __forceinline__ int vertical(int gy) const { return (gy > 0) + (gy < H - 1); }
};

// |d| raises m on its bit pattern (NaN does not).
__device__ __forceinline__ void raise(unsigned long long &m, double d)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(d) & 0x7fffffffffffffffull;
    if (b > m && b <= 0x7ff0000000000000ull) m = b;
}

// Walks the colour's cells of region rows [lo, hi) dealt out over the warps
// in consecutive stretches, calling f(r, q, sum) with the neighbour sum.
template <typename F>
__device__ __forceinline__ void walk(const Block64 &s, int c, int lo, int hi, F f)
{
    lo = max(lo, -s.oy);  // grid rows only
    hi = min(hi, s.H - s.oy);
    const int len = hi - lo;
    if (len <= 0) return;
    // (the two warps of a scheduler take neighbouring stretches, so that the
    // schedulers' shares differ by one row at most)
    const int slot = (s.warp & 3) * (kB64Warps / 4) + (s.warp >> 2);
    const int r0 = lo + len * slot / kB64Warps, r1 = lo + len * (slot + 1) / kB64Warps;
    if (r0 >= r1) return;
    const double *O = s.xrow(1 - c, r0);
    int q = (c + s.oy + r0) & 1;
    double mid = O[0];
    // left + up of the first row (lane 0 and 31 see themselves beyond the
    // region: they are halo or outside the grid)
    double lu = (q ? mid : __shfl_up_sync(0xffffffffu, mid, 1)) + O[-32];
#pragma unroll 2
    for (int r = r0; r < r1; r++, q ^= 1) {
        O += 32;
        const double dn = O[0];
        const double nb = __shfl_down_sync(0xffffffffu, mid, 1);
        const double rd = (q ? nb : mid) + dn;
        f(r, q, lu + rd);
        const double below = __shfl_up_sync(0xffffffffu, rd, 1);
        lu = q ? below : rd;
        mid = dn;
    }
}

template <bool TRACK>
__device__ __forceinline__ void relax64(const Block64 &s, int c, int lo, int hi, double omc, unsigned long long &mx)
{
    walk(s, c, lo, hi, [&](int r, int q, double sum) {
        double *V = s.xrow(c, r);
        const double v = *V;
        const double vn = fma(s.weight(q, s.vertical(s.oy + r)), sum, fma(omc, v, -*s.wbrow(c, r)));
        if (q ? s.act1 : s.act0) *V = vn;
        if (TRACK && (q ? s.own1 : s.own0) && r >= s.h && r < s.h + s.R) raise(mx, vn - v);
    });
}

__global__ void __launch_bounds__(kB64Threads, 1) k_sor_blocks64(Blocks64Args a)
{
    extern __shared__ __align__(16) unsigned char smem_b[];
    __shared__ double s_v[2];
    Block64 s;
    const int g = blockIdx.x, ty = g / a.TX, tx = g - ty * a.TX;
    s.h = 2 * a.K;
    s.H = a.H;
    s.y0 = (int)((long long)ty * a.H / a.TY);
    s.y1 = (int)((long long)(ty + 1) * a.H / a.TY);
    const int WP = (a.W + 1) >> 1;
    s.x0 = 2 * (int)((long long)tx * WP / a.TX);
    s.x1 = min(a.W, 2 * (int)((long long)(tx + 1) * WP / a.TX));
    s.oy = s.y0 - s.h;
    s.ox = s.x0 - s.h;  // x0 and h even: colour of (ox + j, y) is (j + y) & 1
    s.R = s.y1 - s.y0;
    s.RT = s.R + 2 * s.h;
    s.k = threadIdx.x & 31;
    s.warp = threadIdx.x >> 5;
    s.ps = (a.RTmax + 2) * 32;
    s.X = reinterpret_cast<double *>(smem_b);
    s.WB = s.X + 2 * s.ps;
    const int gx0 = s.ox + 2 * s.k, gx1 = gx0 + 1, bl = s.x0 - s.h, br = s.x1 + s.h;
    s.act0 = gx0 >= 0 && gx0 < a.W && gx0 >= bl && gx0 < br;
    s.act1 = gx1 >= 0 && gx1 < a.W && gx1 >= bl && gx1 < br;
    s.own0 = gx0 >= s.x0 && gx0 < s.x1;
    s.own1 = gx1 >= s.x0 && gx1 < s.x1;
    s.cx0 = (gx0 > 0) + (gx0 < a.W - 1);
    s.cx1 = (gx1 > 0) + (gx1 < a.W - 1);
    s.wi0 = a.w64[min(4, s.cx0 + 2)];
    s.wi1 = a.w64[min(4, s.cx1 + 2)];
    s.we0 = a.w64[s.cx0 + 1];
    s.we1 = a.w64[s.cx1 + 1];

    // ---- planes zeroed, then the grid's cells of the region; the places of
    // the halo pairs (row << 8 | lane; a pair's second column may lie outside
    // an odd grid, and then holds 0)
    unsigned *table = reinterpret_cast<unsigned *>(s.WB + 2 * s.ps);
    for (int i = threadIdx.x; i < 4 * s.ps; i += kB64Threads) s.X[i] = 0.0;
    __syncthreads();
    for (int r = s.warp; r < s.RT; r += kB64Warps) {
        const int gy = s.oy + r;
        if (gy < 0 || gy >= a.H) continue;
        const int cy = s.vertical(gy);
#pragma unroll
        for (int q = 0; q < 2; q++) {
            if (!(q ? s.act1 : s.act0)) continue;
            const int c = (q + gy) & 1;
            const size_t i = (size_t)gy * a.ld + gx0 + q;
            *s.xrow(c, r) = a.phi[i];
            *s.wbrow(c, r) = s.weight(q, cy) * a.b[i];
        }
    }
    const int side = s.h / 2;  // halo pairs on each side
    const int np = (s.x1 - s.x0 + 1) / 2;
    const int n_tb = 2 * s.h * kB64Pairs, n_all = n_tb + s.R * 2 * side;
    for (int id = threadIdx.x; id < n_all; id += kB64Threads) {
        int r, k;
        if (id < n_tb) {
            r = id >> 5;
            r = r < s.h ? r : r + s.R;
            k = id & 31;
        } else {
            const int j = id - n_tb;
            r = s.h + j / (2 * side);
            k = j % (2 * side);
            k = k < side ? k : k + np;
        }
        const int gy = s.oy + r, gx = s.ox + 2 * k;
        const bool in = gy >= 0 && gy < a.H && gx >= 0 && gx < a.W && gx >= bl && gx < br;
        table[id] = in ? (unsigned)(r << 8 | k) : ~0u;
    }
    __syncthreads();

    const double omc = 1.0 - a.omega, bnorm = *(volatile const double *)&a.ctl->bnorm;
    const bool track = a.stop == PCD_STOP_MAX_UPDATE, mute = a.withhold && g == 0;
    unsigned ep = 0, checks = 0;
    int sweeps = 0, converged = 0;
    double rel = -1.0, rmax = 0.0, last_max = 0.0;
    unsigned long long mx = 0ull;
    bool failed = false;
    for (;;) {
        // ---- the own cells and the halo hold epoch ep
        if (sweeps > 0 && (sweeps % a.check_every == 0 || sweeps >= a.max_iter)) {
            double acc = 0.0;
            if (!track) {
                mx = 0ull;
#pragma unroll
                for (int c = 0; c < 2; c++)
                    walk(s, c, s.h, s.h + s.R, [&](int r, int q, double sum) {
                        if (!(q ? s.own1 : s.own0)) return;
                        const int gy = s.oy + r, cnt = (q ? s.cx1 : s.cx0) + s.vertical(gy);
                        const double bi = __ldg(a.b + (size_t)gy * a.ld + gx0 + q);
                        const double res = fma((double)cnt, *s.xrow(c, r), bi) - sum;
                        acc = fma(res, res, acc);
                        raise(mx, res);
                    });
            }
            double v[2] = {acc, __longlong_as_double((long long)mx)};
            block_reduce<2, 2u>(v);
            ++checks;
            Words *part = reinterpret_cast<Words *>(a.part) + (size_t)(checks & 1u) * a.G;
            if (threadIdx.x == 0 && !mute) st4(part + g, pack(v[0], v[1], checks));
            // every CTA folds the same partials in the same order: thread t
            // the CTAs t, t + 256, ..., then the block
            double sum = 0.0, most = 0.0;
            for (int t = threadIdx.x; t < a.G; t += kB64Threads) {
                long long it = 0;
                Words p = ld4(part + t);
                while (!failed && !fresh(p, checks)) {
                    if (!again(&a.ctl->error, a.spin_limit, it)) failed = true;
                    p = ld4(part + t);
                }
                sum += first(p);
                most = nan_skip_max(most, second(p));
            }
            double u[2] = {sum, most};
            block_reduce<2, 2u>(u);
            if (threadIdx.x == 0) {
                s_v[0] = u[0];
                s_v[1] = u[1];
            }
            failed = __syncthreads_or(failed);
            if (failed) break;
            if (track) {
                last_max = s_v[1];
                converged = last_max < a.tol;
            } else {
                const double rn = sqrt(s_v[0]);
                rel = bnorm > 0.0 ? rn / bnorm : rn;
                rmax = s_v[1];
                converged = rel <= a.tol;
            }
            if (converged || sweeps >= a.max_iter) break;
            __syncthreads();
        }

        // ---- one round: nsw sweeps, the relaxed rows shrinking with the
        // dependency cone of the own rows
        const int to_check = a.check_every - sweeps % a.check_every;
        const int nsw = min(min(a.K, to_check), a.max_iter - sweeps);
        const bool tested = track && (nsw == to_check || sweeps + nsw >= a.max_iter);
        mx = 0ull;
        for (int t = 0; t < nsw; t++) {
            const int d = 2 * (nsw - t) - 1;
            const bool tr = tested && t == nsw - 1;
            if (tr) relax64<true>(s, 0, s.h - d, s.h + s.R + d, omc, mx);
            else relax64<false>(s, 0, s.h - d, s.h + s.R + d, omc, mx);
            __syncthreads();
            if (tr) relax64<true>(s, 1, s.h - d + 1, s.h + s.R + d - 1, omc, mx);
            else relax64<false>(s, 1, s.h - d + 1, s.h + s.R + d - 1, omc, mx);
            __syncthreads();
        }
        sweeps += nsw;

        // ---- exchange
        ++ep;
        Words *xb = reinterpret_cast<Words *>(a.xb) + (size_t)(ep & 1u) * a.H * WP;
        const int op = s.ox / 2;  // (ox is even)
        if (!mute && s.own0) {
            const int kr = s.k - side;  // the pair's number among the own ones
            const bool edge = (kr < side && tx > 0) || (kr >= np - side && tx < a.TX - 1);
            for (int r = s.h + s.warp; r < s.h + s.R; r += kB64Warps) {
                if (!edge && !(r < 2 * s.h && ty > 0) && !(r >= s.R && ty < a.TY - 1)) continue;
                const int gy = s.oy + r, c = gy & 1;
                st4(xb + (size_t)gy * WP + op + s.k, pack(*s.xrow(c, r), *s.xrow(1 - c, r), ep));
            }
        }
        constexpr int U = 2;
        for (int id0 = threadIdx.x; id0 < n_all; id0 += U * kB64Threads) {
            unsigned at[U];
            bool any = false;
#pragma unroll
            for (int u = 0; u < U; u++) {
                at[u] = id0 + u * kB64Threads < n_all ? table[id0 + u * kB64Threads] : ~0u;
                any = any || at[u] != ~0u;
            }
            long long it = 0;
            while (any && !failed) {
                any = false;
                Words v[U];
#pragma unroll
                for (int u = 0; u < U; u++)
                    if (at[u] != ~0u)
                        v[u] = ld4(xb + (size_t)(s.oy + (int)(at[u] >> 8)) * WP + op + (int)(at[u] & 255u));
#pragma unroll
                for (int u = 0; u < U; u++)
                    if (at[u] != ~0u) {
                        if (fresh(v[u], ep)) {
                            const int r = (int)(at[u] >> 8), k = (int)(at[u] & 255u), c = (s.oy + r) & 1;
                            s.X[c * s.ps + (r + 1) * 32 + k] = first(v[u]);
                            s.X[(1 - c) * s.ps + (r + 1) * 32 + k] = second(v[u]);
                            at[u] = ~0u;
                        } else {
                            any = true;
                        }
                    }
                if (any && !again(&a.ctl->error, a.spin_limit, it)) failed = true;
            }
        }
        failed = __syncthreads_or(failed);
        if (failed) break;
    }
    if (failed) return;  // the error word is set; the solve reports it

    for (int r = s.h + s.warp; r < s.h + s.R; r += kB64Warps) {
        const int gy = s.oy + r;
#pragma unroll
        for (int q = 0; q < 2; q++)
            if (q ? s.own1 : s.own0) a.phi[(size_t)gy * a.ld + gx0 + q] = *s.xrow((q + gy) & 1, r);
    }
    if (g == 0 && threadIdx.x == 0) {
        volatile Ctl *c = a.ctl;
        c->sweeps = sweeps;
        c->converged = converged;
        c->rel = rel;
        c->rmax = rmax;
        c->last_max = last_max;
        c->checks = (int)checks;
        c->halt = 1;
        c->done = 1;
    }
}

}  // namespace

int blocks64_plan(int dev, int W, int H, int K, Blocks64Plan *plan)
{
    if (K < 0 || K > 8 || W < 8 || H < 8) return PCD_BAD_ARG;
    int sms = 0, max_smem = 0, coop = 0;
    PCD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    PCD_CUDA(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    PCD_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    if (!coop) return PCD_BAD_ARG;
    Blocks64Plan best;
    double best_t = 0.0;
    for (int k = K > 0 ? K : 1; k <= (K > 0 ? K : 4); k *= 2) {
        const int h = 2 * k, pairs_max = kB64Pairs - h, WP = (W + 1) / 2;
        if (pairs_max < 1) continue;
        const int TX = (WP + pairs_max - 1) / pairs_max;
        // blocks at least h wide and tall, so the eight neighbours cover the halo
        if (TX > 1 && 2 * (WP / TX) - 1 < h) continue;
        const int TY = std::min(sms / std::max(1, TX), H / h);
        if (TX > sms || TY < 1 || (TY > 1 && H / TY < h) || TX * TY < 2) continue;
        const int n = (H + TY - 1) / TY, RT = n + 2 * h;
        const size_t smem = (size_t)4 * (RT + 2) * 32 * sizeof(double) + ((size_t)2 * h * kB64Pairs + (size_t)n * h) * 4;
        if (smem + 8192 > (size_t)max_smem) continue;
        // us of a sweep: the FP64 pipe's time for the busiest scheduler's rows
        // (4 operations of 64 cycles at 1.9 GHz), each half sweep's barrier and
        // first rows, and an exchange per k sweeps.  Measured with 1, 2 and 4
        // sweeps: 512^2 4.83, 4.36, 4.80; 256^2 2.92, 2.37, 2.51; 252 x 188
        // 2.66, 2.18, 2.33; 64^2 2.24, 1.86, 2.30; 768^2 7.97, 7.93, 8.40.
        const double rows = n + (2 * k - 1);
        const double t = 2.0 * (((int)(rows / 4.0 + 0.99)) * 0.135 + 0.25) + 1.6 / k;
        if (!best.K || t < best_t) {
            best_t = t;
            best.TY = TY;
            best.TX = TX;
            best.K = k;
            best.RTmax = RT;
            best.smem = smem;
            best.xb_bytes = (size_t)2 * H * WP * 32;
        }
    }
    if (!best.K) return PCD_BAD_ARG;
    PCD_CUDA(allow_shared((const void *)k_sor_blocks64));
    *plan = best;
    return PCD_OK;
}

int launch_blocks64(Blocks64Args &a, const Blocks64Plan &p, cudaStream_t s)
{
    a.TY = p.TY;
    a.TX = p.TX;
    a.G = p.TY * p.TX;
    a.K = p.K;
    a.RTmax = p.RTmax;
    void *params[] = {&a};
    PCD_CUDA(cudaLaunchCooperativeKernel((const void *)k_sor_blocks64, dim3(a.G), dim3(kB64Threads), params, p.smem, s));
    count_launches(1);
    return PCD_OK;
}

}  // namespace pcd
