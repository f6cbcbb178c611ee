// sor_resident.cu -- FP32 red-black SOR sweeps of the correction equation
// L e = r32 with the whole grid resident on the chip (sm_103a).
//
// The grid is cut into TX x TY tiles, one CTA each, all co-resident
// (cooperative launch).  A CTA holds its tile plus a halo of 2K cells on every
// side that has a neighbour; e lives in registers for the whole launch, -r32 in
// shared memory.
// K sweeps run between two exchanges: the dependency cone of K red-black
// sweeps ends inside the halo, whose values are recomputed with the owner's
// arithmetic and thrown away at the next exchange.
//
// The lanes' part of a tile is sor_tile.cuh's, the exchange's words those of
// words.cuh, double-buffered by epoch parity: a CTA overwrites epoch n's word
// with epoch n + 2 only after it read its neighbours' epoch n + 1, which they
// publish after reading epoch n.
//
// Two ways to end a launch:
//   cycle   an FP32 estimate of ||r32 - L e|| every check_every sweeps, its
//           partials (tagged words as above) read one round later, so that
//           their trip overlaps the sweeps; the cycle ends `lag` sweeps after
//           the estimate that passed, from a copy of e written then where the
//           round has gone further;
//   chunk   exactly nsw sweeps.  With the max-update stop every tracked
//           sweep's largest |update| goes to a global maximum; after the last
//           sweep one grid barrier makes them visible, and if an earlier sweep
//           already passed the test the chunk runs again from e = 0 up to that
//           sweep (once a solve), so no sweep ever waits for the test.
//
// Bound: latency.  At 512^2 (6 x 25 tiles of 88 x 22 cells, K = 8, 14 warps) a
// sweep takes 0.62-0.67 us against the one-cluster form's 2.08 (16 SMs,
// sor_cluster_rr.cuh): 16 half sweeps of about 470 cycles (64 instructions a
// warp; shuffle, edge row, five dependent packed operations, block barrier)
// and about 2900 cycles of exchange a round; 1.15-1.2 us at 1024^2 against
// 5.7 of the tile passes of that time.  Measured on the way: a separate update
// for the border rows set the pace of the
// grid (0.72 against 0.59 us on one tile); 16-byte exchange accesses fetch
// each sector twice (1.48 against 1.15 us a sweep at 1024^2); publishing each
// colour as it becomes final gains nothing.
#include <algorithm>

#include "sor_resident.cuh"
#include "sor_tile.cuh"
#include "words.cuh"

namespace pcd {

namespace {

using namespace tile;
using namespace words;

__device__ __forceinline__ unsigned rs_ld_acquire(const unsigned *p)
{
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ Quad rs_quad(const Words &v)
{
    return {make_float2(__uint_as_float((unsigned)v.x), __uint_as_float((unsigned)v.y)),
            make_float2(__uint_as_float((unsigned)v.z), __uint_as_float((unsigned)v.w))};
}

__device__ __forceinline__ Words rs_words(const Quad &q, unsigned ep)
{
    return {word(__float_as_uint(q.a.x), ep), word(__float_as_uint(q.a.y), ep), word(__float_as_uint(q.b.x), ep),
            word(__float_as_uint(q.b.y), ep)};
}

// Most warps of a CTA: as few as the tiles need, for the registers that L rows
// of both colours take (512 threads of 128 registers spill from L = 4 on).
__host__ __device__ constexpr int rs_warps(int L) { return L == 2 ? 16 : 12; }

// Shared memory of a CTA: the tile's, the landing planes of the halo quads (the
// -r32 planes' shape, only halo places written) and the table of the halo quads.
// halo quads of a tile with n own rows: the rows above and below, then the
// lane columns left and right of the own rows
__host__ __device__ inline int rs_halo_quads(int K, int CL, int n)
{
    return 4 * (2 * K) * CL + n * 4 * (K / 4);
}
inline size_t rs_smem(int K, int L, int CL, int NG, int n, bool exchange)
{
    size_t b = (edge_quads(CL, NG) + plane_quads(L, CL, NG)) * sizeof(Quad);
    if (exchange) b += plane_quads(L, CL, NG) * sizeof(Quad) + (size_t)rs_halo_quads(K, CL, n) * sizeof(uint2);
    return b;
}

template <int K, int L, int CL, bool RAG>
__global__ void __launch_bounds__(32 * rs_warps(L), 1) k_sor_resident(ResidentArgs a)
{
    using T = Tile<L, CL, RAG>;
    constexpr int HK = 2 * K, HL = HK / 8;  // halo rows, halo lane columns
    static_assert(K % 4 == 0, "the halo is a whole number of lane columns");
    extern __shared__ __align__(16) float smem_f[];
    __shared__ float s_red[32];
    __shared__ float s_vals[kResidentCtasMax];
    __shared__ float s_tot;
    __shared__ double s_lim;  // squared estimate that ends the cycle
    __shared__ unsigned s_mx[kResidentChecksMax];
    __shared__ int s_first;
    Ctl *ctl = a.ctl;
    {
        const volatile Ctl *c = ctl;
        if (c->halt || c->done || c->error || c->nan_cells) return;  // every CTA reads the same
    }
    const int done_before = ((volatile const Ctl *)ctl)->sweeps;
    const int target0 = min(a.nsw, a.max_iter - done_before);
    if (target0 < 1) return;

    // ---- the tile and the lane's part of it
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, NW = blockDim.x >> 5, NT = blockDim.x;
    const int G = gridDim.x, g = blockIdx.x, ty = g / a.TX, tx = g - ty * a.TX;
    const int H2 = (a.H + 1) >> 1;  // tiles start on even rows
    const int yb = 2 * (int)((long long)ty * H2 / a.TY), ye = min(a.H, 2 * (int)((long long)(ty + 1) * H2 / a.TY));
    const int qb = (int)((long long)tx * a.KQ / a.TX), qe = (int)((long long)(tx + 1) * a.KQ / a.TX);
    const int hr = a.TY > 1 ? HK : 0, hl = a.TX > 1 ? HL : 0;
    const int n = ye - yb, nq = qe - qb, R = n + 2 * hr;
    const int ybase = yb - hr, qbase = qb - hl;

    T st;
    st.place(smem_f, a.NG);
    st.y0 = ybase + st.lr0;
    const int q = qbase + st.cl;
    const bool act = st.cl < nq + 2 * hl && q >= 0 && q < a.KQ;
    st.own = st.cl >= hl && st.cl < hl + nq;
    st.zl = q == 0;
    st.nvalid = min(8, a.W - 8 * q);
    st.zr = q == a.KQ - 1 && st.nvalid == 8;
    st.H = a.H;
    st.setup_weights(act, R, a.w32);
    st.gin = st.y0 < a.H && st.y0 + L > 0;
    st.brd = __any_sync(0xffffffffu, st.gin && (st.y0 <= 0 || st.y0 + L >= a.H));
    for (unsigned z = threadIdx.x; z < edge_quads(CL, a.NG); z += NT) reinterpret_cast<Quad *>(smem_f)[z] = quad_zero();
    Quad *rp = reinterpret_cast<Quad *>(smem_f) + edge_quads(CL, a.NG);
    Quad *land = rp + plane_quads(L, CL, a.NG);
    uint2 *table = reinterpret_cast<uint2 *>(land + plane_quads(L, CL, a.NG));
    constexpr unsigned grow = 16u * CL;  // bytes of a plane's row
    // the lane's place in the landing planes, which are one of each colour
    const unsigned land_s = st.r_s + 2u * st.r_c;
    const unsigned xplane = (unsigned)a.H * (unsigned)a.KQ;  // exchange quads of one colour
    // rows of the lane that go out (pub) and come in (imp) at an exchange
    unsigned pub = 0, imp = 0;
    int halo_quads = 0;
    if (G > 1) {
#pragma unroll
        for (int j = 0; j < L; j++) {
            const int lr = st.lr0 + j, y = st.y0 + j;
            const bool mine = st.own && lr >= hr && lr < hr + n;
            const bool border = (lr < hr + HK && ty > 0) || (lr >= hr + n - HK && ty < a.TY - 1) ||
                                (st.cl < 2 * hl && tx > 0) || (st.cl >= nq && tx < a.TX - 1);
            if (mine && border && !(a.withhold && g == 0)) pub |= 1u << j;
            if (!mine && act && lr < R && y >= 0 && y < a.H) imp |= 1u << j;
        }
        // every halo quad's exchange word and landing place, dealt out over
        // the threads (the lanes that own the side columns would have 2 L
        // serial loads each); outside the grid: ~0
        halo_quads = rs_halo_quads(K, CL, n);
        for (int id = threadIdx.x; id < halo_quads; id += NT) {
            constexpr int nt = 4 * HK * CL;
            int lr, cc, c;
            if (id < nt) {
                const int r = id / CL;
                cc = id & (CL - 1);
                c = r & 1;
                lr = (r >> 1) < HK ? (r >> 1) : (r >> 1) + n;
            } else {
                const int k = id - nt, sd = k & (2 * HL - 1), r = k / (2 * HL);
                cc = sd < HL ? sd : nq + sd;
                c = r & 1;
                lr = hr + (r >> 1);
            }
            const int y = ybase + lr, qq = qbase + cc;
            const bool in = y >= 0 && y < a.H && qq >= 0 && qq < a.KQ && cc < nq + 2 * hl &&
                            (id < nt ? a.TY > 1 : a.TX > 1);
            table[id] = in ? make_uint2((unsigned)c * xplane + (unsigned)y * (unsigned)a.KQ + (unsigned)qq,
                                        (unsigned)((c * a.NG * L + lr) * CL + cc))
                           : make_uint2(~0u, 0u);
        }
    }

    // ---- -r32 of the tile and its halo; e = 0
#pragma unroll
    for (int j = 0; j < L; j++) {
        const int lr = st.lr0 + j, y = st.y0 + j;
        const bool in = lr < R && y >= 0 && y < a.H && act;
        st.copy_row(st.r_s, j, a.r32 + (in ? (long)y * 8 * a.KQ : 0), q, a.KQ, in);
    }
    st.copies_wait();
    const double bnorm = ((volatile const Ctl *)ctl)->bnorm;
    const double rstart = ((volatile const Ctl *)ctl)->rnorm;
    if (threadIdx.x == 0) {
        const double stop_abs = kFp32StopFrac * a.tol * bnorm, drop_abs = a.drop * rstart;
        s_lim = fmax(stop_abs * stop_abs, drop_abs * drop_abs);
    }
    unsigned ep = ((volatile const Ctl *)ctl)->res_epoch;     // exchanges so far
    unsigned ck = ((volatile const Ctl *)ctl)->res_checks;    // estimates so far

    // the tile's own rows of e to global memory
    auto store_own = [&]() {
#pragma unroll
        for (int j = 0; j < L; j++) {
            const int lr = st.lr0 + j, y = st.y0 + j;
            if (!st.own || lr < hr || lr >= hr + n) continue;
            st.store_row(j, a.e + (long)y * 8 * a.KQ, q, a.KQ);
        }
    };

    const bool track0 = a.gran > 0;
    if (track0)
        for (int t = threadIdx.x; t < kResidentChecksMax; t += NT) s_mx[t] = 0u;

    int sweeps = 0, target = target0, passed = -1;
    bool track = track0, failed = false, saved = false;
    float last_max = 0.f;
    for (int phase = 0;; phase++) {
#pragma unroll
        for (int j = 0; j < L; j++) st.e[0][j] = st.e[1][j] = quad_zero();
        st.template put_edges<0>();
        st.template put_edges<1>();
        __syncthreads();
        sweeps = 0;
        int next_check = a.cycle ? (a.check_every + a.dep - 1) / a.dep * a.dep : 0x7fffffff;
        int snap_at = -1, next_tr = a.gran;
        bool pending = false, to_post = false, est_now = false;
        for (;;) {
            if (est_now) {
                // an estimate of the state at `sweeps`; its partials wait in
                // s_red for the next block barrier
                float v = st.residual(hr, hr + n);
                v = warp_sum_f(v);
                if (lane == 0) s_red[w] = v;
                est_now = false;
                to_post = pending = true;
                ++ck;
                snap_at = sweeps + a.lag;
                if (a.lag == 0) store_own();
            }
            const int kr = min(K, min(target, next_check) - sweeps);
            // half sweep i relaxes the rows within 2 kr - 1 - i of the tile's
            // own (the dependency cone); a warp further out sits it out.  The
            // other rows outside the cone are relaxed along, and overwritten
            // at the next exchange.
            const int live = 2 * kr - 1 - max(hr - st.whi, st.wlo - hr - n);
            // stretches of plain sweeps, cut where something else is due
            for (int t = 0; t < kr;) {
                const int s0 = sweeps + t;
                if (track && (s0 + 1 == next_tr || s0 + 1 == target)) {
                    float mx = 0.f;
                    if (2 * t < live) st.template half<0, true>(mx, hr, hr + n);
                    __syncthreads();
                    if (2 * t + 1 < live) st.template half<1, true>(mx, hr, hr + n);
                    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                    if (lane == 0 && mx > 0.f) atomicMax(&s_mx[s0 / a.gran], __float_as_uint(mx));
                    __syncthreads();
                    if (s0 + 1 == next_tr) next_tr += a.gran;
                    t++;
                    continue;
                }
                int end = to_post ? t + 1 : kr;
                if (track) end = min(end, min(next_tr, target) - 1 - sweeps);
                if (snap_at > s0) end = min(end, snap_at - sweeps);
                float none = 0.f;
                int i = 2 * t;
#pragma unroll 1
                do {
                    if (i < live) st.template half<0, false>(none, 0, 0);
                    __syncthreads();
                    if (i + 1 < live) st.template half<1, false>(none, 0, 0);
                    __syncthreads();
                    i += 2;
                } while (i < 2 * end);
                t = end;
                if (to_post) {
                    if (w == 0) {
                        float x = lane < NW ? s_red[lane] : 0.f;
                        x = warp_sum_f(x);
                        if (lane == 0) {
                            if (G == 1) s_tot = x;
                            else if (!(a.withhold && g == 0)) st1(a.part + (size_t)(ck & 1) * G + g, word(__float_as_uint(x), ck));
                        }
                    }
                    to_post = false;
                }
                if (sweeps + t == snap_at && a.lag > 0 && t < kr) store_own();
            }
            sweeps += kr;
            const bool last = sweeps >= target;
            const bool decide = pending && sweeps >= snap_at;
            // (the border quads leave before anything is waited for, and the
            // partials below are polled while they travel: 1.92 ms a 512^2 solve,
            // with the poll first and one warp's sum behind a barrier 1.96)
            Words *xb = nullptr;
            if (!last && G > 1) {
                ++ep;
                xb = reinterpret_cast<Words *>(a.xb) + (size_t)(ep & 1) * 2 * xplane;
                // ---- own border quads out
                if (pub) {
                    Words *p = xb + ((long)st.y0 * a.KQ + q);
#pragma unroll
                    for (int j = 0; j < L; j++, p += a.KQ)
                        if (pub >> j & 1u) {
                            st4(p, rs_words(st.e[0][j], ep));
                            st4(p + xplane, rs_words(st.e[1][j], ep));
                        }
                }
            }
            if (decide && G > 1) {
                // the partials of every CTA, posted at least half a sweep ago
                for (int t = threadIdx.x; t < G; t += NT) {
                    const unsigned long long *p = a.part + (size_t)(ck & 1) * G + t;
                    long long it = 0;
                    unsigned long long v = ld1(p);
                    while ((unsigned)(v >> 32) != ck && !failed) {
                        if (!again(&a.ctl->error, a.spin_limit, it)) failed = true;
                        v = ld1(p);
                    }
                    s_vals[t] = __uint_as_float((unsigned)v);
                }
            }
            if (!last && G > 1) {
                // ---- halo quads in
                constexpr int U = L <= 4 ? 4 : 2;
                for (int id0 = threadIdx.x; id0 < halo_quads; id0 += U * NT) {
                    uint2 at[U];
                    bool any = false;
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        at[u] = id0 + u * NT < halo_quads ? table[id0 + u * NT] : make_uint2(~0u, 0u);
                        any = any || at[u].x != ~0u;
                    }
                    long long it = 0;
                    while (any && !failed) {
                        any = false;
                        Words v[U];
#pragma unroll
                        for (int u = 0; u < U; u++)
                            if (at[u].x != ~0u) v[u] = ld4(xb + at[u].x);
#pragma unroll
                        for (int u = 0; u < U; u++)
                            if (at[u].x != ~0u) {
                                if (fresh(v[u], ep)) {
                                    land[at[u].y] = rs_quad(v[u]);
                                    at[u].x = ~0u;
                                } else {
                                    any = true;
                                }
                            }
                        if (any && !again(&a.ctl->error, a.spin_limit, it)) failed = true;
                    }
                }
                __syncthreads();
                if (imp) {
#pragma unroll
                    for (int j = 0; j < L; j++)
                        if (imp >> j & 1u) {
                            st.e[0][j] = ldsq(land_s + grow * (unsigned)j);
                            st.e[1][j] = ldsq(land_s + st.r_c + grow * (unsigned)j);
                        }
                }
                st.template put_edges<0>();
                st.template put_edges<1>();
            }
            if (G > 1 ? __syncthreads_or(failed) : 0) { failed = true; break; }
            if (decide) {
                float tot;
                if (G > 1) {
                    // every warp of every CTA sums the same partials in the same order
                    float x = 0.f;
                    for (int t = lane; t < G; t += 32) x += s_vals[t];
                    tot = warp_sum_f(x);
                } else {
                    __syncthreads();  // (posted behind the last sweep's barrier)
                    tot = s_tot;
                }
                pending = false;
                const double est2 = (double)tot;
                if (est2 <= s_lim) {
                    if (sweeps > snap_at) saved = true;  // e of sweep snap_at was written then
                    sweeps = snap_at;
                    break;
                }
            }
            if (last) break;
            if (sweeps >= next_check) {
                est_now = true;
                next_check = (sweeps + a.check_every + a.dep - 1) / a.dep * a.dep;
            }
        }
        if (failed || !track) break;
        // ---- max-update stop: the first tracked sweep that passed
        const int np = (target - 1) / a.gran + 1;
        __syncthreads();
        for (int t = threadIdx.x; t < np; t += NT)
            if (s_mx[t]) atomicMax(&a.gmax[t], s_mx[t]);
        if (threadIdx.x == 0) s_first = np;
        __syncthreads();
        if (G > 1) {
            if (threadIdx.x == 0 && !(a.withhold && g == 0)) {
                __threadfence();
                atomicAdd(a.bar, 1u);
            }
            if (threadIdx.x == 0) {
                long long it = 0;
                while (rs_ld_acquire(a.bar) < (unsigned)G && !failed)
                    if (!again(&a.ctl->error, a.spin_limit, it)) failed = true;
            }
            if (__syncthreads_or(failed)) { failed = true; break; }
        } else {
            __threadfence();
            __syncthreads();
        }
        for (int t = threadIdx.x; t < np; t += NT)
            if ((double)__uint_as_float(__ldcg(a.gmax + t)) < a.tol) atomicMin(&s_first, t);
        __syncthreads();
        const int first = s_first;
        last_max = __uint_as_float(__ldcg(a.gmax + min(first, np - 1)));
        if (first < np) {
            passed = min((first + 1) * a.gran, target);
            if (passed < target) {
                target = passed;
                track = false;
                continue;  // once more from e = 0, up to the sweep that passed
            }
        }
        break;
    }
    if (failed) return;  // the error word is set; the solve reports it
    if (!saved) store_own();
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&ctl->blocks_done, 1u) == gridDim.x - 1) {
            volatile Ctl *c = ctl;
            const int s = done_before + sweeps;
            c->sweeps = s;
            if (track0) {
                c->last_max = (double)last_max;
                if (passed >= 0) {
                    c->converged = 1;
                    c->halt = 1;
                }
                const int np = (target0 - 1) / a.gran + 1;
                for (int t = 0; t < np; t++) ((volatile unsigned *)a.gmax)[t] = 0u;
                *(volatile unsigned *)a.bar = 0u;
            }
            if (s >= a.max_iter) c->halt = 1;
            c->res_epoch = ep;
            c->res_checks = ck;
            c->blocks_done = 0;
            __threadfence();
        }
    }
}

template <int K, bool RAG>
const void *rs_kernel_l(int L, int CL)
{
    if (CL == 8) return K == 4 && L == 2 ? (const void *)k_sor_resident<4, 2, 8, RAG> : nullptr;
    if (CL != 16) return nullptr;
    switch (L) {
    case 2: return (const void *)k_sor_resident<K, 2, 16, RAG>;
    case 4: return (const void *)k_sor_resident<K, 4, 16, RAG>;
    }
    if constexpr (!RAG) {
        // (partial lane columns need twice the weight registers)
        switch (L) {
        case 6: return (const void *)k_sor_resident<K, 6, 16, RAG>;
        case 8: return (const void *)k_sor_resident<K, 8, 16, RAG>;
        }
    }
    return nullptr;
}

const void *rs_kernel(int K, int L, int CL, bool rag)
{
    if (K == 4) return rag ? rs_kernel_l<4, true>(L, CL) : rs_kernel_l<4, false>(L, CL);
    if (K == 8) return rag ? rs_kernel_l<8, true>(L, CL) : rs_kernel_l<8, false>(L, CL);
    return nullptr;
}

}  // namespace

int resident_plan(int dev, int W, int H, ResidentPlan *plan)
{
    if (W < 16 || H < 16) return PCD_BAD_ARG;
    int sms = 0, max_smem = 0, coop = 0;
    PCD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    PCD_CUDA(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    PCD_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    if (!coop) return PCD_BAD_ARG;
    sms = std::min(sms, kResidentCtasMax);
    const int KQ = (W + 7) / 8, H2 = (H + 1) / 2;
    ResidentPlan best;
    double best_t = 0.0;
    for (int K : {4, 8})
        for (int CL : {8, 16})
            for (int L : {2, 4, 6, 8}) {
                if (!rs_kernel(K, L, CL, W % 8 != 0)) continue;
                const int G = 32 / CL, HK = 2 * K, HL = HK / 8;
                for (int TX = 1; TX <= std::min(sms, KQ); TX++) {
                    const int nq = (KQ + TX - 1) / TX;
                    if (nq + (TX > 1 ? 2 * HL : 0) > CL) continue;
                    if (TX > 1 && KQ / TX < HL) break;
                    // most tile rows whose tiles hold a neighbour's whole halo
                    int tymax = sms / TX;
                    while (tymax > 1 && 2 * (H2 / tymax) - H % 2 < HK) tymax--;
                    for (int TY : {tymax, 1}) {
                        const int n = std::min(H, 2 * ((H2 + TY - 1) / TY)), R = n + (TY > 1 ? 2 * HK : 0);
                        const int NW = std::max(4, ((R + L - 1) / L + G - 1) / G), NG = NW * G;
                        if (NW > rs_warps(L)) continue;
                        const size_t smem = rs_smem(K, L, CL, NG, n, TX * TY > 1);
                        if (smem + 8192 > (size_t)max_smem) continue;
                        // ns of a sweep.  Without exchanges (one-tile grids,
                        // 1, 2 and 3 warps a scheduler) it measured, L = 2:
                        // 284, 376, 468; L = 4: 362, 504, 650; L = 6: 546,
                        // 760, 1027; L = 8: 796, 1007, 1270.  An exchange
                        // measured 1.2-1.4 us with L = 2 and 1.8-2.3 us
                        // above; warps outside the cone save 10-15%.
                        const int wps = (NW + 3) / 4;
                        double t = (L == 2 ? 284 : L == 4 ? 362 : L == 6 ? 546 : 796) +
                                   (wps - 1) * (L == 2 ? 92 : L == 4 ? 144 : 240);
                        if (TX * TY > 1) t = (K == 8 ? 0.85 : 0.9) * t + (L == 2 ? 1300.0 : 2000.0) / K;
                        if (best.L == 0 || t < best_t) {
                            best_t = t;
                            best.K = K;
                            best.L = L;
                            best.CL = CL;
                            best.TX = TX;
                            best.TY = TY;
                            best.NW = NW;
                            best.NG = NG;
                            best.R = R;
                            best.KQ = KQ;
                            best.smem = smem;
                            best.xb_bytes = TX * TY > 1 ? (size_t)4 * H * KQ * 32 : 0;
                        }
                    }
                }
            }
    if (!best.L) return PCD_BAD_ARG;
    // (here and not in front of every launch, which it would hold up)
    PCD_CUDA(allow_shared(rs_kernel(best.K, best.L, best.CL, W % 8 != 0)));
    *plan = best;
    return PCD_OK;
}

int launch_resident(ResidentArgs &a, const ResidentPlan &p, cudaStream_t s)
{
    const void *fn = rs_kernel(p.K, p.L, p.CL, a.W % 8 != 0);
    if (!fn) {
        set_error("resident SOR: no kernel for this plan");
        return PCD_BAD_ARG;
    }
    a.KQ = p.KQ;
    a.TX = p.TX;
    a.TY = p.TY;
    a.NG = p.NG;
    a.R = p.R;
    void *params[] = {&a};
    if (p.TX * p.TY == 1) PCD_CUDA(cudaLaunchKernel(fn, dim3(1), dim3(32 * p.NW), params, p.smem, s));
    else PCD_CUDA(cudaLaunchCooperativeKernel(fn, dim3(p.TX * p.TY), dim3(32 * p.NW), params, p.smem, s));
    count_launches(1);
    return PCD_OK;
}

}  // namespace pcd
