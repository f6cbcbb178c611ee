// sor_tile.cu -- FP32 red-black SOR passes over grids that live in HBM (sm_103a):
// up to four sweeps of the correction equation L e = r32 per pass, from one
// buffer into the other, each tile of the grid held in registers for the pass.
//
// At 4096 x 4096 a sweep takes 10.6 us (25.8 when every pass was a launch whose
// warps loaded 16-row tiles before they swept them, 12.4 when it was a launch of
// these tiles), at 2048 x 1500 2.5 us (5.3; 3.9); with an FP64 refresh every 512
// sweeps 11.1 and 2.65.  A tile takes 3.3 us, of which its
// eight half sweeps take 2.5: 38% of issue slots busy, three warps a scheduler
// that wait for one another's edge rows.  On grids of two or three tiles a CTA
// the way of a halo through L2 (store, report, poll, load) comes on top.
//
// Tiles of up to 96 rows x 16 lane columns (128 cells), halo included: tile
// (ty, tx) writes the rows [ty N, ty N + N), N <= 96 - 2 hk even, hk = 2 x the
// sweeps of a pass, and the lane columns [qb, qe), one lane column (eight cells) of halo on
// each side; the written parts partition the grid.  The relaxed rows shrink
// with the dependency cone of the written ones; columns are all relaxed in
// every half sweep, and the wrong value that enters at a tile's outer column
// spreads by one cell a half sweep, eight cells a pass at most.
//
// One persistent CTA per SM takes the tiles of pass after pass in row-major
// order, so that tiles in flight share their halo rows through L2.  12 warps
// sweep; while they are on one tile a producer warp has TMA bring the next one's
// correction and right-hand side into shared memory and a storing warp has it
// write the last one's correction (edge rows, three pairs of planes and the
// written rows: 212 KB).  Tiles wait for their neighbours' previous pass, not
// for all of it.  With TRACK every pass reports the largest |update| of its last
// sweep.
//
// k_tile_batch runs the same tiles for many grids at once: the grids' tiles are
// numbered one after the other (TileJob::tile0), and the CTAs stride over all
// of them, skipping the grids whose solves have halted.
#include <algorithm>
#include <string>

#include "sor_passes.cuh"
#include "sor_tile.cuh"
#include "tensor_map.cuh"
#include "words.cuh"

namespace pcd {

namespace {

using namespace tile;

constexpr int kTL = 4, kTCL = 16, kTWarps = 12, kTThreads = 32 * kTWarps;
// A fourth warpgroup, with the producer and the storing warp, lends the sweeping ones
// registers: 512 x 128 at launch = 384 x 152 + 128 x 56.
constexpr int kTBlock = kTThreads + 128, kTRegsSweep = 152, kTRegsProduce = 56;
static_assert(kTThreads * kTRegsSweep + 128 * kTRegsProduce <= kTBlock * 128, "registers of the launch");

constexpr int kTGroups = kTWarps * (32 / kTCL), kTRows = kTGroups * kTL;  // 96
// RAG: the form with every cell's own weights, for the last tile column of a grid
// whose last lane column is not whole, or also the first (8 cells wide).
// UNI: a tile all of whose rows have both vertical neighbours.
template <bool RAG, bool UNI>
using TileT = Tile<kTL, kTCL, RAG, UNI>;
inline bool ragged(int W) { return W % 8 != 0 || W == 8; }

// edge rows, two sets of -r32 planes (this tile's and the next one's), the next
// tile's correction; and the written part of the last tile's (the written lane
// columns of its written rows, a row of each plane)
constexpr size_t kTQuads = (size_t)4 * (kTGroups + 1) * kTCL + (size_t)3 * 2 * kTGroups * kTL * kTCL;
constexpr int kTOutRow = kTCL - 2, kTOutRows = kTRows - 8;
constexpr size_t kTOutQuads = (size_t)2 * kTOutRow * kTOutRows;
inline size_t tile_smem() { return (kTQuads + kTOutQuads) * sizeof(Quad); }
constexpr unsigned kTPlaneBytes = 2u * kTGroups * kTL * kTCL * (unsigned)sizeof(Quad);

// Where tile t of a W x H grid lies.
struct TileGeom {
    int ybase, n;     // first loaded row, written rows
    int qbase, nq;    // first loaded lane column, written lane columns
};

__device__ __forceinline__ TileGeom tile_geom(int t, int ncol, int N, int KQ, int H, int hk)
{
    const int ty = t / ncol, tx = t - ty * ncol;
    TileGeom g;
    const int nq = KQ / ncol, extra = KQ - nq * ncol;  // the first `extra` tile columns are one wider
    g.qbase = tx * nq + min(tx, extra) - 1;
    g.nq = nq + (tx < extra);
    g.ybase = ty * N - hk;
    g.n = min(N, H - ty * N);
    return g;
}

// A tile of a pass, as the producer warp hands it to the sweeping ones.
struct TileItem {
    TileGeom g;
    int job;    // of a batch
    int kr;     // sweeps; 0: no more tiles, -1: a wait gave up
    int first;  // the correction starts at 0
    int side;   // reads ea (0) or eb, writes the other
    int wide;   // one of the wider tile columns
    int pass;
    int tile;   // in done[]
    unsigned epoch;  // its value there once the tile is in memory
};

// What the warps of a CTA share.  Phase n of each mbarrier belongs to the CTA's
// tile n, whose item is item[n & 3].
struct TileShared {
    unsigned long long full;     // the tile has landed
    unsigned long long free;     // its correction has left the landing planes
    unsigned long long staged;   // its new correction is in the output rows
    unsigned long long drained;  // it has left them
    TileItem item[4];
};

__device__ __forceinline__ unsigned shared_at(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned bar, int count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect(unsigned bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ void mbar_arrive(unsigned bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// Waits for phase `parity` of an mbarrier, two seconds at most; false on
// timeout.
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity)
{
    constexpr unsigned kNs = 1000;
    for (int i = 0; i < (1 << 21); i++) {
        unsigned ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity), "r"(kNs)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// Barrier of the sweeping warps.
__device__ __forceinline__ void sweep_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kTThreads) : "memory"); }
__device__ __forceinline__ bool sweep_sync_or(bool v)
{
    unsigned r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "bar.red.or.pred q, 1, %2, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((unsigned)v), "n"(kTThreads)
        : "memory");
    return r;
}

__device__ __forceinline__ void tile_box(unsigned to, const CUtensorMap *map, const TileGeom &g, int plane, unsigned bar)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(to), "l"(map), "r"(4 * g.qbase), "r"(plane), "r"(g.ybase), "r"(bar)
        : "memory");
}

// Starts the copies of a tile, one thread: the correction (ein; nullptr: it
// starts at 0) into the landing planes, -r32 into plane set `set`; zeros where
// a box leaves the grid.  Four boxes of up to 96 rows x 256 bytes.  (cp.async
// by every lane held all warps at the load unit for 2100 of a tile's 7000
// cycles; a 256-byte bulk copy a row from 384 threads for 2400 to 4000.)
__device__ __forceinline__ void tile_fetch(const void *smem, const TileGeom &g, const CUtensorMap *ein,
                                           const CUtensorMap *r32, int rows, int set, unsigned bar)
{
    mbar_expect(bar, (unsigned)rows * (2u * kTCL * (unsigned)sizeof(Quad)) * (ein ? 2u : 1u));
    const unsigned planes = shared_at(smem) + (unsigned)(edge_quads(kTCL, kTGroups) * sizeof(Quad));
    for (int s = 0; s < 2; s++) {
        const unsigned to = planes + (unsigned)s * (kTPlaneBytes / 2);
        if (ein) tile_box(to + 2u * kTPlaneBytes, ein, g, s, bar);
        tile_box(to + (unsigned)set * kTPlaneBytes, r32, g, s, bar);
    }
}

// The producer warp: hands out the CTA's tiles, each when the tiles that it
// depends on are in memory.  Tile t of pass p reads and overwrites what its up
// to eight neighbours wrote and read in pass p - 1, so it waits for their and
// its own done[] to reach base + p; the CTAs pass no barrier between passes.
// Every CTA takes its tiles in the order of (p, t), so the lowest unfinished
// tile never waits for an unfinished one.  Tile n is fetched while the sweeping
// warps are on tile n - 1.
//   next(it, nb): the CTA's next tile, false at the end; nb: the lane's
//   neighbour in done[] (-1: none); start(it, n): its copies
template <typename Next, typename Start>
__device__ __forceinline__ void tile_produce(TileShared *sh, const unsigned *done, unsigned base, int *error,
                                             long long limit, Next next, Start start)
{
    const int lane = threadIdx.x & 31;
    const unsigned full = shared_at(&sh->full), free_ = shared_at(&sh->free);
    bool ok = true, more = true;
    for (int n = 0; ok && more; n++) {
        TileItem it{};
        int nb = -1;
        more = next(it, nb);
        if (more && it.pass > 0) {
            long long polls = 0;
            bool mine = nb < 0;
            while (ok && !mine) {
                unsigned v;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(done + nb) : "memory");
                mine = (int)(v - (base + (unsigned)it.pass)) >= 0;
                if (!mine) ok = words::again(error, limit, polls);
            }
            ok = __all_sync(0xffffffffu, ok);
            __syncwarp();
            asm volatile("fence.proxy.async;" ::: "memory");
        }
        // (before a failure is handed on, too: a phase takes one arrival)
        if (n > 0) ok = __all_sync(0xffffffffu, mbar_wait(free_, (n - 1) & 1)) && ok;
        if (lane == 0) {
            if (!more || !ok) it.kr = ok ? 0 : -1;
            it.epoch = base + (unsigned)it.pass + 1u;
            sh->item[n & 3] = it;
            if (it.kr > 0) start(it, n);
            else mbar_arrive(full);
            if (!ok) atomicCAS(error, 0, PCD_TIMEOUT);
        }
        __syncwarp();
    }
}

// The storing warp: copies a tile's staged rows to memory (a box of each plane)
// and then reports the tile done.  (Stored by the sweeping warps, a tile held
// each for 900 cycles, and the fence in front of its report took 3200; a bulk
// copy a row took twice the time of the sweeps.)
//   grid(it): the map of the tile's output buffer
template <typename Grid>
__device__ __forceinline__ void tile_drain(const void *smem, TileShared *sh, int hk, unsigned *done, int *error,
                                           int withhold, Grid grid)
{
    if ((threadIdx.x & 31) != 0) return;
    const unsigned from = shared_at(smem) + (unsigned)(kTQuads * sizeof(Quad));
    for (int n = 0;; n++) {
        if (!mbar_wait(shared_at(&sh->staged), n & 1)) {
            atomicCAS(error, 0, PCD_TIMEOUT);
            return;
        }
        const TileItem it = sh->item[n & 3];
        if (it.kr <= 0) return;
        const CUtensorMap *map = grid(it);
        for (int s = 0; s < 2; s++)
            asm volatile(
                "cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3}], [%4];" ::"l"(map),
                "r"(4 * (it.g.qbase + 1)), "r"(s), "r"(it.g.ybase + hk),
                "r"(from + (unsigned)s * (unsigned)(kTOutQuads / 2 * sizeof(Quad)))
                : "memory");
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        mbar_arrive(shared_at(&sh->drained));
        asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");  // (the copies are visible to this thread)
        if (!(withhold && it.tile == 0))
            asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(done + it.tile), "r"(it.epoch) : "memory");
    }
}

// kr <= hk / 2 sweeps on the tile in the landing planes and plane set `set`.
template <bool TRACK, bool RAG, bool UNI>
__device__ __forceinline__ bool tile_sweeps(float *smem, TileShared *sh, const TileItem &it, int W, int H, int hk,
                                            int n, const float *w32, float &mx)
{
    const TileGeom g = it.g;
    const int kr = it.kr;
    TileT<RAG, UNI> st;
    st.place(smem, kTGroups);
    const int q = g.qbase + st.cl, KQ = (W + 7) >> 3;
    const bool act = st.cl < g.nq + 2 && q >= 0 && q < KQ;
    st.y0 = g.ybase + st.lr0;
    st.H = H;
    st.own = st.cl >= 1 && st.cl <= g.nq;
    st.zl = q == 0;
    st.nvalid = RAG ? min(8, W - 8 * q) : 8;
    st.zr = q == KQ - 1 && st.nvalid == 8;
    st.gin = st.y0 < H && st.y0 + kTL > 0;
    st.brd = __any_sync(0xffffffffu, st.gin && (st.y0 <= 0 || st.y0 + kTL >= H));
    st.setup_weights(act, kTRows, w32);
    const unsigned land = st.r_s + 2u * kTPlaneBytes;
    st.r_s += (unsigned)(n & 1) * kTPlaneBytes;
#pragma unroll
    for (int j = 0; j < kTL; j++)
#pragma unroll
        for (int c = 0; c < 2; c++) st.e[c][j] = it.first ? quad_zero() : ldsq(st.plane_at(land, c, j));
    st.template put_edges<0>();
    st.template put_edges<1>();
    sweep_sync();
    if (threadIdx.x == 0) mbar_arrive(shared_at(&sh->free));
    const int live = 2 * kr - 1 - max(hk - st.whi, st.wlo - hk - g.n);
    float none = 0.f;
#pragma unroll 1
    for (int i = 0; i < 2 * (TRACK ? kr - 1 : kr); i += 2) {
        if (i < live) st.template half<0, false>(none, 0, 0);
        sweep_sync();
        if (i + 1 < live) st.template half<1, false>(none, 0, 0);
        sweep_sync();
    }
    if (TRACK) {
        if (2 * kr - 2 < live) st.template half<0, true>(mx, hk, hk + g.n);
        sweep_sync();
        if (2 * kr - 1 < live) st.template half<1, true>(mx, hk, hk + g.n);
    }
    if (n > 0 && !__all_sync(0xffffffffu, mbar_wait(shared_at(&sh->drained), (n - 1) & 1))) return false;
    const unsigned out = shared_at(smem) + (unsigned)(kTQuads * sizeof(Quad));
#pragma unroll
    for (int j = 0; j < kTL; j++) {
        const int r = st.lr0 + j - hk;
        if (st.own && r >= 0 && r < g.n)
#pragma unroll
            for (int c = 0; c < 2; c++)
                stsq(out + (unsigned)(((c ^ j) & 1) * (int)(kTOutQuads / 2) + r * g.nq + st.cl - 1) * (unsigned)sizeof(Quad),
                     st.e[c][j]);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(shared_at(&sh->staged));
    return true;
}

// The sweeping warps: tile after tile, as they land.  grid(it, W, H, w32): the
// grid of a tile; gmax: each pass's largest |update| (TRACK).
template <bool TRACK, bool RAGGED, typename Grid>
__device__ __forceinline__ void tile_consume(float *smem, TileShared *sh, int hk, int *error, unsigned *gmax, Grid grid)
{
    const unsigned full = shared_at(&sh->full);
    bool fine = true;
    for (int n = 0;; n++) {
        fine = __all_sync(0xffffffffu, fine && mbar_wait(full, n & 1));
        // (the previous tile's half sweeps are done with the edge rows, too)
        if (sweep_sync_or(!fine)) {
            mbar_wait(full, n & 1);  // (no copy of ours outlives the CTA)
            if (threadIdx.x == 0) atomicCAS(error, 0, PCD_TIMEOUT);
            return;
        }
        const TileItem it = sh->item[n & 3];
        if (it.kr <= 0) {
            // the storing warp ends, too: one phase, which may not complete before
            // that warp has seen the last tile's
            if (n > 0) mbar_wait(shared_at(&sh->drained), (n - 1) & 1);
            __syncwarp();
            if ((threadIdx.x & 31) == 0) mbar_arrive(shared_at(&sh->staged));
            return;
        }
        const float *w32;
        int W, H;
        grid(it, W, H, w32);
        float mx = 0.f;
        if (RAGGED && it.g.qbase + it.g.nq + 2 >= (W + 7) >> 3)
            fine = tile_sweeps<TRACK, RAGGED, false>(smem, sh, it, W, H, hk, n, w32, mx);
        else if (it.g.ybase > 0 && it.g.ybase + kTRows < H)
            fine = tile_sweeps<TRACK, false, true>(smem, sh, it, W, H, hk, n, w32, mx);
        else
            fine = tile_sweeps<TRACK, false, false>(smem, sh, it, W, H, hk, n, w32, mx);
        if (TRACK) {
            const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(mx));
            if ((threadIdx.x & 31) == 0 && m) atomicMax(gmax + it.pass, m);
        }
    }
}

__device__ __forceinline__ void tile_begin(float *smem, TileShared *sh)
{
    // (the rows above the first and below the last group are never published,
    // and rows past a box are never written: finite numbers there)
    for (unsigned z = threadIdx.x; z < kTQuads; z += kTBlock) reinterpret_cast<Quad *>(smem)[z] = quad_zero();
    if (threadIdx.x == 0) {
        mbar_init(shared_at(&sh->full), 1);
        mbar_init(shared_at(&sh->free), 1);
        mbar_init(shared_at(&sh->staged), kTWarps);
        mbar_init(shared_at(&sh->drained), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
}

// The lane's neighbour (itself included) of tile t = (ty, tx), or -1.
__device__ __forceinline__ int tile_neighbour(int t, int ncol, int nrow)
{
    const int lane = threadIdx.x & 31, ty = t / ncol + lane / 3 - 1, tx = t % ncol + lane % 3 - 1;
    return lane < 9 && ty >= 0 && ty < nrow && tx >= 0 && tx < ncol ? ty * ncol + tx : -1;
}

// `sweeps` sweeps from 0 in ea, nsw in a pass (fewer in the last one and at the
// sweep cap).  TRACK: the max-update stop, after every pass or (!each) after the
// launch's last one.  Where a pass that is
// not the launch's last one meets it, the launch has run too far: it leaves the
// sweeps up to that pass in ctl->redo, and a launch with `again` (one without
// TRACK) runs these, the first time's bits.
template <bool TRACK, bool RAGGED>
__global__ void __launch_bounds__(kTBlock, 1)
    k_tile_pass(const __grid_constant__ TileMaps maps, Ctl *ctl, unsigned *done, const __grid_constant__ SolveArgs a, int ncol, int nrow, int N, int hk, int nsw,
                int sweeps, int again, int each, unsigned *gmax, long long limit, int withhold)
{
    if (*(volatile const int *)&ctl->halt || *(volatile const int *)&ctl->error) return;
    const int total = again ? *(volatile const int *)&ctl->redo
                            : min(sweeps, a.max_iter - *(volatile const int *)&ctl->sweeps);
    if (total < 1) return;  // every CTA reads the same count
    extern __shared__ __align__(128) float smem_f[];  // (TMA boxes start at 128-byte addresses)
    __shared__ TileShared sh;
    tile_begin(smem_f, &sh);
    const unsigned base = *(volatile const unsigned *)&ctl->res_epoch;
    const int ntiles = ncol * nrow, KQ = (a.W + 7) >> 3, passes = (total + nsw - 1) / nsw;
    if (threadIdx.x >= kTThreads) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kTRegsProduce));
        const int role = ((int)threadIdx.x - kTThreads) >> 5;
        int t = (int)blockIdx.x - (int)gridDim.x, p = 0;
        if (role == 0) tile_produce(
            &sh, done, base, &ctl->error, limit,
            [&](TileItem &it, int &nb) {
                t += gridDim.x;
                while (t >= ntiles) {
                    t -= ntiles;
                    p++;
                }
                if (p >= passes) return false;
                it.g = tile_geom(t, ncol, N, KQ, a.H, hk);
                it.kr = min(nsw, total - p * nsw);
                it.first = p == 0;
                it.side = p & 1;
                it.wide = it.g.nq > KQ / ncol;
                it.pass = p;
                it.tile = t;
                nb = tile_neighbour(t, ncol, nrow);
                return true;
            },
            [&](const TileItem &it, int n) {
                tile_fetch(smem_f, it.g, it.first ? nullptr : &maps.in[it.side], &maps.r32, N + 2 * hk,
                           n & 1, shared_at(&sh.full));
            });
        else if (role == 1) tile_drain(smem_f, &sh, hk, done, &ctl->error, withhold,
                                       [&](const TileItem &it) { return &maps.out[it.side ? 0 : 1][it.wide]; });
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kTRegsSweep));
        tile_consume<TRACK, RAGGED>(smem_f, &sh, hk, &ctl->error, gmax,
                                    [&](const TileItem &, int &W, int &H, const float *&w32) {
                                        W = a.W;
                                        H = a.H;
                                        w32 = a.w32;
                                    });
    }
    __shared__ bool s_last;
    __shared__ int s_first;
    __syncthreads();
    if (threadIdx.x == 0) {
        s_first = passes;
        __threadfence();
        s_last = atomicAdd(&ctl->blocks_done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    if (TRACK) {
        for (int p = (each ? 0 : passes - 1) + (int)threadIdx.x; p < passes; p += kTBlock)
            if ((double)__uint_as_float(__ldcg(gmax + p)) < a.tol) atomicMin(&s_first, p);
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        volatile Ctl *c = ctl;
        if (TRACK) c->last_max = (double)__uint_as_float(__ldcg(gmax + min(s_first, passes - 1)));
        c->stream_out = passes & 1;
        c->res_epoch = base + (unsigned)passes;
        c->blocks_done = 0;
        c->redo = 0;
        if (TRACK && s_first < passes - 1) {
            c->redo = (s_first + 1) * nsw;
        } else {
            const int n = c->sweeps + total;
            c->sweeps = n;
            if (again || (TRACK && s_first < passes)) c->converged = 1;
            if (again || (TRACK && s_first < passes) || n >= a.max_iter) c->halt = 1;
        }
    }
    if (TRACK) {
        __syncthreads();
        for (int p = threadIdx.x; p < passes; p += kTBlock) gmax[p] = 0u;
    }
}

// The job owning global tile `t` (tile0 ascending from 0).
__device__ __forceinline__ int tile_job(const int *tile0, int njobs, int t)
{
    int lo = 0, hi = njobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (tile0[mid] <= t) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Written rows of a tile of an H-row grid in a batch.
__host__ __device__ inline int batch_rows(int H)
{
    const int most = kTRows - 4 * kTilePassSweeps;
    return H < most ? (H + 1) & ~1 : most;
}

// Up to `sweeps` sweeps over the tiles of every job (grid) of a batch whose
// solve has not halted, in passes of four from ea into eb and back, the
// corrections starting from 0.  Each CTA
// keeps every job's first tile and its sweeps for this launch in shared memory,
// the latter from its control block at the start (the blocks change only at
// the end of the launch); the CTA that finishes last closes it for every
// job that ran (sweep count, sweep cap, ping-pong side) and resets the counter.
// sync: finished CTAs, epoch of done[].
template <bool RAGGED>
__global__ void __launch_bounds__(kTBlock, 1)
    k_tile_batch(const TileJob *__restrict__ jobs, int njobs, int ntiles, int sweeps, unsigned *sync, unsigned *done,
                 long long limit, int withhold)
{
    constexpr int hk = 2 * kTilePassSweeps;
    extern __shared__ __align__(128) float smem_f[];  // (TMA boxes start at 128-byte addresses)
    __shared__ TileShared sh;
    __shared__ bool s_last;
    int *s_tile0 = reinterpret_cast<int *>(reinterpret_cast<Quad *>(smem_f) + kTQuads + kTOutQuads),
        *s_total = s_tile0 + njobs;
    // the batch's error word is the first grid's
    int *error = &jobs[0].ctl->error;
    if (__syncthreads_or(threadIdx.x == 0 && *(volatile const int *)error)) return;
    for (int j = threadIdx.x; j < njobs; j += kTBlock) {
        const TileJob &J = jobs[j];
        const volatile Ctl *c = J.ctl;
        s_tile0[j] = J.tile0;
        s_total[j] = c->halt ? 0 : max(0, min(sweeps, J.max_iter - c->sweeps));
    }
    tile_begin(smem_f, &sh);
    // (the host wrote the jobs' maps to global memory: a thread for each tile of
    // the CTA makes its grid's maps visible to the copies)
    for (int t = blockIdx.x + threadIdx.x * gridDim.x; t < ntiles; t += kTBlock * gridDim.x) {
        const TileMaps &m = jobs[tile_job(s_tile0, njobs, t)].maps;
        for (const CUtensorMap *map = &m.in[0]; map != &m.in[0] + sizeof(TileMaps) / sizeof(CUtensorMap); map++)
            asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(map) : "memory");
    }
    __syncthreads();
    const unsigned base = *(volatile const unsigned *)(sync + 1);
    const int passes = (sweeps + kTilePassSweeps - 1) / kTilePassSweeps;
    if (threadIdx.x >= kTThreads) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kTRegsProduce));
        const int role = ((int)threadIdx.x - kTThreads) >> 5;
        int t = (int)blockIdx.x - (int)gridDim.x, p = 0;
        if (role == 0) tile_produce(
            &sh, done, base, error, limit,
            [&](TileItem &it, int &nb) {
                for (;;) {
                    t += gridDim.x;
                    while (t >= ntiles) {
                        t -= ntiles;
                        p++;
                    }
                    if (p >= passes) return false;
                    it.job = tile_job(s_tile0, njobs, t);
                    it.kr = min(kTilePassSweeps, s_total[it.job] - kTilePassSweeps * p);
                    if (it.kr > 0) break;
                }
                const TileJob &J = jobs[it.job];
                it.g = tile_geom(t - J.tile0, J.ncol, batch_rows(J.H), J.W >> 3, J.H, hk);
                it.first = p == 0;
                it.side = p & 1;
                it.wide = it.g.nq > (J.W >> 3) / J.ncol;
                it.pass = p;
                it.tile = t;
                nb = tile_neighbour(t - J.tile0, J.ncol, J.nrow);
                if (nb >= 0) nb += J.tile0;
                return true;
            },
            [&](const TileItem &it, int n) {
                const TileJob &J = jobs[it.job];
                tile_fetch(smem_f, it.g, it.first ? nullptr : &J.maps.in[it.side], &J.maps.r32,
                           batch_rows(J.H) + 2 * hk, n & 1, shared_at(&sh.full));
            });
        else if (role == 1) tile_drain(smem_f, &sh, hk, done, error, withhold,
                                       [&](const TileItem &it) { return &jobs[it.job].maps.out[it.side ? 0 : 1][it.wide]; });
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kTRegsSweep));
        tile_consume<false, RAGGED>(smem_f, &sh, hk, error, nullptr,
                                    [&](const TileItem &it, int &W, int &H, const float *&w32) {
                                        const TileJob &J = jobs[it.job];
                                        W = J.W;
                                        H = J.H;
                                        w32 = J.w32;
                                    });
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(sync, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (s_last) {
        __threadfence();
        // (tiles were left out where a wait gave up: no grid's corrections are
        // whole, and the refresh, which sees the word too, folds none of them in)
        if (*(volatile const int *)error) return;
        for (int j = threadIdx.x; j < njobs; j += kTBlock) {
            if (s_total[j] < 1) continue;
            volatile Ctl *c = jobs[j].ctl;
            c->stream_out = ((s_total[j] + kTilePassSweeps - 1) / kTilePassSweeps) & 1;
            const int sw = c->sweeps + s_total[j];
            c->sweeps = sw;
            if (sw >= jobs[j].max_iter) c->halt = 1;
        }
        if (threadIdx.x == 0) {
            sync[0] = 0u;
            sync[1] = base + (unsigned)passes;
        }
        __threadfence();
    }
}

const void *tile_kernel(bool track, bool rag)
{
    if (rag) return track ? (const void *)k_tile_pass<true, true> : (const void *)k_tile_pass<false, true>;
    return track ? (const void *)k_tile_pass<true, false> : (const void *)k_tile_pass<false, false>;
}

const void *batch_kernel(bool narrow)
{
    return narrow ? (const void *)k_tile_batch<true> : (const void *)k_tile_batch<false>;
}

}  // namespace

int tile_plan(int dev, int W, int H, int depth, TilePlan *plan)
{
    if (W < 8 || H < 1) return PCD_BAD_ARG;
    if (depth != 0 && depth != 2 && depth != 4) return PCD_BAD_ARG;
    TilePlan p;
    p.K = depth ? depth : kTilePassSweeps;
    p.ncol = ceil_div(ceil_div(W, 8), kTCL - 2);
    p.nrow = ceil_div(H, kTRows - 4 * p.K);
    p.smem = tile_smem();
    int sms = 0, bps = 0;
    PCD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    for (bool track : {false, true}) {
        const void *fn = tile_kernel(track, ragged(W));
        PCD_CUDA(allow_shared(fn));
        PCD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, fn, kTBlock, p.smem));
        if (bps < 1) return PCD_BAD_ARG;
    }
    // The tallest tiles recompute the fewest halo rows, and passes that no barrier
    // parts have no last round of CTAs to fill (with a refresh every 512 sweeps,
    // 2048 x 1500: 361 tiles of 80 rows 2.65 us a sweep, 456 of 64 rows, three full
    // rounds, 3.66; 2048^2 3.03 and 3.56).  Grids that leave SMs idle are cut finer.
    const long most = (long)sms * bps, tiles = (long)p.ncol * p.nrow, rounds = (tiles + most - 1) / most;
    if (rounds == 1)
        p.nrow = (int)std::max<long>(p.nrow, std::min<long>(rounds * most / p.ncol, ceil_div(H, 16)));
    p.rows = 2 * ceil_div(H, 2L * p.nrow);
    p.nrow = ceil_div(H, p.rows);
    p.grid = (int)std::min<long>((long)p.ncol * p.nrow, most);
    *plan = p;
    return PCD_OK;
}

int tile_maps(float *ea, float *eb, const float *r32, int W, int H, int ncol, int rows, int halo, TileMaps *m)
{
    const auto fn = tensor_map_encoder();
    if (!fn) {
        set_error("tile SOR: cuTensorMapEncodeTiled is not available");
        return PCD_DEVICE_ERROR;
    }
    const cuuint64_t KQ = ((cuuint64_t)W + 7) / 8;
    const cuuint64_t dims[3] = {4 * KQ, 2, (cuuint64_t)H}, strides[2] = {16 * KQ, 32 * KQ};
    auto encode = [&](CUtensorMap *map, const float *base, int quads, int box_rows) {
        const cuuint32_t box[3] = {4 * (cuuint32_t)quads, 1, (cuuint32_t)box_rows}, estr[3] = {1, 1, 1};
        const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float *>(base), dims, strides, box,
                              estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r == CUDA_SUCCESS) return (int)PCD_OK;
        set_error("tile SOR: cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")");
        return (int)PCD_DEVICE_ERROR;
    };
    const int nq = (int)KQ / ncol, wide = (int)KQ % ncol ? 1 : 0;
    float *const e[2] = {ea, eb};
    for (int i = 0; i < 2; i++) {
        PCD_TRY(encode(&m->in[i], e[i], kTCL, rows + 2 * halo));
        for (int w = 0; w < 2; w++) PCD_TRY(encode(&m->out[i][w], e[i], nq + (w & wide), rows));
    }
    return encode(&m->r32, r32, kTCL, rows + 2 * halo);
}

int launch_tile(const TilePlan &p, const TileMaps &maps, Ctl *ctl, unsigned *done, unsigned *gmax, const SolveArgs &a,
                int nsw, int sweeps, bool each, long long limit, int withhold, cudaStream_t s)
{
    if (nsw < 1 || nsw > p.K || sweeps < 1) {
        set_error("tile SOR: more sweeps than the plan's halo holds");
        return PCD_BAD_ARG;
    }
    const bool track = a.stop == PCD_STOP_MAX_UPDATE;
    int ncol = p.ncol, nrow = p.nrow, rows = p.rows, hk = 2 * p.K, again = 0, every = each ? 1 : 0;
    void *params[] = {const_cast<TileMaps *>(&maps), &ctl, &done, const_cast<SolveArgs *>(&a), &ncol, &nrow, &rows, &hk,
                      &nsw, &sweeps, &again, &every, &gmax, &limit, &withhold};
    PCD_CUDA(cudaLaunchCooperativeKernel(tile_kernel(track, ragged(a.W)), dim3(p.grid), dim3(kTBlock), params, p.smem, s));
    count_launches(1);
    if (track && each && sweeps > nsw) {
        again = 1;
        PCD_CUDA(cudaLaunchCooperativeKernel(tile_kernel(false, ragged(a.W)), dim3(p.grid), dim3(kTBlock), params, p.smem,
                                             s));
        count_launches(1);
    }
    return PCD_OK;
}

int tile_job_setup(TileJob *job)
{
    job->ncol = ceil_div(job->W / 8, kTCL - 2);
    job->nrow = ceil_div(job->H, batch_rows(job->H));
    return tile_maps(job->ea, job->eb, job->r32, job->W, job->H, job->ncol, batch_rows(job->H), 2 * kTilePassSweeps,
                     &job->maps);
}

int tile_batch_config(int dev, int njobs, bool narrow, size_t *smem, int *grid)
{
    if (njobs < 1 || njobs > kTileBatchJobsMax) {
        set_error("batched tile pass: 1 to " + std::to_string(kTileBatchJobsMax) + " grids");
        return PCD_BAD_ARG;
    }
    const void *fn = batch_kernel(narrow);
    const size_t per_job = 2 * sizeof(int);
    const size_t bytes = tile_smem() + (size_t)njobs * per_job;
    int sms = 0, bps = 0;
    PCD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    PCD_CUDA(allow_shared(fn));
    PCD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, fn, kTBlock, bytes));
    if (bps < 1) {
        set_error("batched tile pass: the kernel does not fit on an SM");
        return PCD_BAD_ARG;
    }
    *smem = bytes;
    *grid = sms * bps;
    return PCD_OK;
}

int launch_tile_batch(const TileJob *d_jobs, int njobs, int ntiles, int sweeps, bool narrow, int grid, size_t smem,
                      unsigned *sync, unsigned *done, long long limit, int withhold, cudaStream_t s)
{
    if (njobs < 1 || njobs > kTileBatchJobsMax || ntiles < 1 || sweeps < 1) {
        set_error("batched tile pass: bad arguments");
        return PCD_BAD_ARG;
    }
    void *params[] = {&d_jobs, &njobs, &ntiles, &sweeps, &sync, &done, &limit, &withhold};
    PCD_CUDA(cudaLaunchCooperativeKernel(batch_kernel(narrow), dim3(std::min(grid, ntiles)), dim3(kTBlock), params, smem,
                                         s));
    return PCD_OK;
}

}  // namespace pcd
