// sor_tile.cu -- FP32 red-black SOR passes over grids that live in HBM (sm_103a):
// up to four sweeps of the correction equation L e = r32 per pass, from one
// buffer into the other, each tile of the grid held in registers for the pass.
//
// At 4096 x 4096, four sweeps a pass: 52.6 us a pass with its refreshes, 94 us
// when warps took 16-row tiles from one another and loaded them before they
// swept; 2048 x 1500: 16.5 us, before 21.  A tile takes 3.4 us, of which its
// eight half sweeps take 2.5 (38% of issue slots busy: three warps a scheduler
// wait for one another's edge rows), the launch and first load 6.5 us a pass.
//
// Tiles of up to 96 rows x 16 lane columns (128 cells), halo included: tile
// (ty, tx) writes the rows [ty N, ty N + N), N <= 96 - 2 hk even, hk = 2 x the
// sweeps of a pass, and the lane columns [qb, qe), one lane column (eight cells) of halo on
// each side; the written parts partition the grid.  The relaxed rows shrink
// with the dependency cone of the written ones; columns are all relaxed in
// every half sweep, and the wrong value that enters at a tile's outer column
// spreads by one cell a half sweep, eight cells a pass at most.
//
// One persistent CTA of 12 warps per SM takes the tiles in row-major order, so
// that tiles in flight share their halo rows through L2; while it sweeps one
// tile, TMA brings the next one's correction and right-hand side into
// shared memory (edge rows and three pairs of planes: 173 KB).  The
// CTA that finishes last closes the pass; with TRACK the pass reports the
// largest |update| of its last sweep.
//
// k_tile_batch runs the same tiles for many grids at once: the grids' tiles are
// numbered one after the other (TileJob::tile0), and the CTAs stride over all
// of them, skipping the grids whose solves have halted.
#include <algorithm>
#include <string>

#include "sor_passes.cuh"
#include "sor_tile.cuh"
#include "tensor_map.cuh"

namespace pcd {

namespace {

using namespace tile;

constexpr int kTL = 4, kTCL = 16, kTWarps = 12, kTThreads = 32 * kTWarps;
constexpr int kTGroups = kTWarps * (32 / kTCL), kTRows = kTGroups * kTL;  // 96
// NARROW: one lane column wide (8 cells), whose lane has both the grid's first
// and its last column; the form with every cell's own weights.
// UNI: a tile all of whose rows have both vertical neighbours.
template <bool NARROW, bool UNI>
using TileT = Tile<kTL, kTCL, NARROW, UNI>;

// edge rows, two sets of -r32 planes (this tile's and the next one's), and the
// next tile's correction
constexpr size_t kTQuads = (size_t)4 * (kTGroups + 1) * kTCL + (size_t)3 * 2 * kTGroups * kTL * kTCL;
inline size_t tile_smem() { return kTQuads * sizeof(Quad); }
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

// One grid's buffers and size in a pass.
struct TileGrid {
    const CUtensorMap *ein;    // nullptr: the correction starts at 0
    float *eout;
    const CUtensorMap *r32;
    int W, H;
};

// ---- a tile's data by TMA, completion on an mbarrier
__device__ __forceinline__ void mbar_init(unsigned bar)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect(unsigned bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// Bounded wait for phase `parity` of an mbarrier; false on timeout.
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity)
{
    for (int i = 0; i < (1 << 22); i++) {
        unsigned ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

__device__ __forceinline__ void tile_box(unsigned to, const CUtensorMap *map, const TileGeom &g, int plane, unsigned bar)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(to), "l"(map), "r"(4 * g.qbase), "r"(plane), "r"(g.ybase), "r"(bar)
        : "memory");
}

// Starts the copies of a tile, one thread: the correction into the landing
// planes, -r32 into plane set `set`; zeros where a box leaves the grid.  Four
// boxes of up to 96 rows x 256 bytes.  (cp.async by every lane held all warps
// at the load unit for 2100 of a tile's 7000 cycles; a 256-byte bulk copy a
// row from 384 threads for 2400 to 4000.)
__device__ __forceinline__ void tile_fetch(const void *smem, const TileGeom &g, const TileGrid &d, int rows, int set,
                                           unsigned bar)
{
    mbar_expect(bar, (unsigned)rows * (2u * kTCL * (unsigned)sizeof(Quad)) * (d.ein ? 2u : 1u));
    const unsigned planes = (unsigned)__cvta_generic_to_shared(smem) +
                            (unsigned)(edge_quads(kTCL, kTGroups) * sizeof(Quad));
    for (int s = 0; s < 2; s++) {
        const unsigned to = planes + (unsigned)s * (kTPlaneBytes / 2);
        if (d.ein) tile_box(to + 2u * kTPlaneBytes, d.ein, g, s, bar);
        tile_box(to + (unsigned)set * kTPlaneBytes, d.r32, g, s, bar);
    }
}

// kr <= hk / 2 sweeps on the tile that tile_fetch asked for (its copies complete
// phase `parity` of bar); next() starts the copies of the one after it,
// once this tile's landing planes have been read.  False when the
// wait gave up.
template <bool TRACK, bool NARROW, bool UNI, typename Next>
__device__ __forceinline__ bool tile_sweeps(float *smem, const TileGeom &g, const TileGrid &d, int hk, int kr, int set,
                                            unsigned bar, unsigned parity, const float *w32, float &mx, Next next)
{
    TileT<NARROW, UNI> st;
    st.place(smem, kTGroups);
    const int q = g.qbase + st.cl, KQ = d.W >> 3, H = d.H;
    const bool act = st.cl < g.nq + 2 && q >= 0 && q < KQ;
    st.y0 = g.ybase + st.lr0;
    st.H = H;
    st.own = st.cl >= 1 && st.cl <= g.nq;
    st.zl = q == 0;
    st.zr = q == KQ - 1;
    st.nvalid = 8;
    st.gin = st.y0 < H && st.y0 + kTL > 0;
    st.brd = __any_sync(0xffffffffu, st.gin && (st.y0 <= 0 || st.y0 + kTL >= H));
    st.setup_weights(act, kTRows, w32);
    const unsigned land = st.r_s + 2u * kTPlaneBytes;
    st.r_s += set * kTPlaneBytes;
    const bool landed = mbar_wait(bar, parity);
#pragma unroll
    for (int j = 0; j < kTL; j++)
#pragma unroll
        for (int c = 0; c < 2; c++)
            st.e[c][j] = d.ein ? ldsq(st.plane_at(land, c, j)) : quad_zero();
    // the previous tile's half sweeps are done with the edge rows, and this
    // tile's correction is in registers
    if (__syncthreads_or(!landed)) {
        mbar_wait(bar, parity);  // (no copy of ours outlives the CTA)
        return false;
    }
    st.template put_edges<0>();
    st.template put_edges<1>();
    __syncthreads();
    const int live = 2 * kr - 1 - max(hk - st.whi, st.wlo - hk - g.n);
    float none = 0.f;
    next();
#pragma unroll 1
    for (int i = 0; i < 2 * (TRACK ? kr - 1 : kr); i += 2) {
        if (i < live) st.template half<0, false>(none, 0, 0);
        __syncthreads();
        if (i + 1 < live) st.template half<1, false>(none, 0, 0);
        __syncthreads();
    }
    if (TRACK) {
        if (2 * kr - 2 < live) st.template half<0, true>(mx, hk, hk + g.n);
        __syncthreads();
        if (2 * kr - 1 < live) st.template half<1, true>(mx, hk, hk + g.n);
    }
#pragma unroll
    for (int j = 0; j < kTL; j++) {
        const int lr = st.lr0 + j;
        if (st.own && lr >= hk && lr < hk + g.n) st.store_row(j, d.eout + (long)(st.y0 + j) * 8 * KQ, q, KQ);
    }
    return true;
}

template <bool TRACK, bool NARROW, typename Next>
__device__ __forceinline__ bool tile_run(float *smem, const TileGeom &g, const TileGrid &d, int hk, int kr, int n,
                                         unsigned bar, const float *w32, float &mx, Next next)
{
    // n: the CTA's tiles before this one
    if (!NARROW && g.ybase > 0 && g.ybase + kTRows < d.H)
        return tile_sweeps<TRACK, NARROW, true>(smem, g, d, hk, kr, n & 1, bar, n & 1, w32, mx, next);
    return tile_sweeps<TRACK, NARROW, false>(smem, g, d, hk, kr, n & 1, bar, n & 1, w32, mx, next);
}

__device__ __forceinline__ void tile_begin(float *smem, unsigned bar)
{
    // (the rows above the first and below the last group are never published,
    // and the copies leave places outside the grid alone: finite numbers there)
    for (unsigned z = threadIdx.x; z < kTQuads; z += kTThreads) reinterpret_cast<Quad *>(smem)[z] = quad_zero();
    if (threadIdx.x == 0) mbar_init(bar);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
}

template <bool TRACK, bool NARROW>
__global__ void __launch_bounds__(kTThreads, 1)
    k_tile_pass(const __grid_constant__ CUtensorMap ein, float *__restrict__ eout,
                const __grid_constant__ CUtensorMap r32, Ctl *ctl, SolveArgs a, int ncol, int nrow, int N, int hk, int nsw, int out_idx, int zero)
{
    if (*(volatile const int *)&ctl->halt || *(volatile const int *)&ctl->error) return;
    const int kr = min(nsw, a.max_iter - *(volatile const int *)&ctl->sweeps);
    if (kr < 1) return;  // every CTA reads the same count
    extern __shared__ __align__(128) float smem_f[];  // (TMA boxes start at 128-byte addresses)
    __shared__ __align__(8) unsigned long long s_bar;
    const unsigned bar = (unsigned)__cvta_generic_to_shared(&s_bar);
    tile_begin(smem_f, bar);
    float mx = 0.f;
    const int ntiles = ncol * nrow, KQ = a.W >> 3;
    const TileGrid d = {zero ? nullptr : &ein, eout, &r32, a.W, a.H};
    auto fetch = [&](int t, int set) {
        if (t < ntiles && threadIdx.x == 0)
            tile_fetch(smem_f, tile_geom(t, ncol, N, KQ, a.H, hk), d, N + 2 * hk, set, bar);
    };
    fetch(blockIdx.x, 0);
    int n = 0;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x, n++)
        if (!tile_run<TRACK, NARROW>(smem_f, tile_geom(t, ncol, N, KQ, a.H, hk), d, hk, kr, n, bar, a.w32, mx,
                                     [&]() { fetch(t + (int)gridDim.x, (n + 1) & 1); })) {
            if (threadIdx.x == 0) atomicCAS(&ctl->error, 0, PCD_TIMEOUT);
            break;
        }
    if (TRACK) {
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        if ((threadIdx.x & 31) == 0 && mx > 0.f)
            atomicMax(&ctl->maxbits, (unsigned long long)__double_as_longlong((double)mx));
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&ctl->blocks_done, 1u) == gridDim.x - 1) {
            __threadfence();
            ((volatile Ctl *)ctl)->stream_out = out_idx;
            end_of_sweep(ctl, a, kr);
        }
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

// One pass of up to nsw sweeps over the tiles of every job (grid) of a batch
// whose solve has not halted: pass parity `par` reads buffer ea (par 0) or
// eb and writes the other; zero: the corrections start from 0.  Each CTA
// keeps every job's first tile and its sweeps for this pass in shared memory,
// the latter from its control block at the start (the blocks change only at
// the end of the pass); the CTA that finishes last closes the pass of every
// job that ran (sweep count, sweep cap, ping-pong side) and resets `counter`.
template <bool NARROW>
__global__ void __launch_bounds__(kTThreads, 1)
    k_tile_batch(const TileJob *__restrict__ jobs, int njobs, int ntiles, int nsw, int par, int zero,
                 unsigned *counter)
{
    constexpr int hk = 2 * kTilePassSweeps;
    extern __shared__ __align__(128) float smem_f[];  // (TMA boxes start at 128-byte addresses)
    __shared__ bool s_last;
    int *s_tile0 = reinterpret_cast<int *>(reinterpret_cast<Quad *>(smem_f) + kTQuads), *s_kr = s_tile0 + njobs;
    for (int j = threadIdx.x; j < njobs; j += kTThreads) {
        const TileJob &J = jobs[j];
        const volatile Ctl *c = J.ctl;
        s_tile0[j] = J.tile0;
        s_kr[j] = c->halt || c->error ? 0 : max(0, min(nsw, J.max_iter - c->sweeps));
    }
    __shared__ __align__(8) unsigned long long s_bar;
    const unsigned bar = (unsigned)__cvta_generic_to_shared(&s_bar);
    tile_begin(smem_f, bar);
    float mx = 0.f;
    auto grid_of = [&](const TileJob &J) {
        return TileGrid{zero ? nullptr : par ? &J.maps.eb : &J.maps.ea, par ? J.ea : J.eb, &J.maps.r32, J.W, J.H};
    };
    auto geom_of = [&](const TileJob &J, int t) {
        return tile_geom(t - J.tile0, J.ncol, batch_rows(J.H), J.W >> 3, J.H, hk);
    };
    // (the host wrote the jobs' maps to global memory: a thread for each tile of
    // the CTA makes its grid's maps visible to the copies)
    for (int t = blockIdx.x + threadIdx.x * gridDim.x; t < ntiles; t += kTThreads * gridDim.x) {
        const TileMaps &m = jobs[tile_job(s_tile0, njobs, t)].maps;
        for (const CUtensorMap *map : {&m.ea, &m.eb, &m.r32})
            asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(map) : "memory");
    }
    __syncthreads();
    // the first tile from t on of a grid that runs
    auto running = [&](int t) {
        while (t < ntiles && s_kr[tile_job(s_tile0, njobs, t)] < 1) t += gridDim.x;
        return t;
    };
    auto fetch = [&](int t, int set) {
        if (t >= ntiles || threadIdx.x != 0) return;
        const TileJob &J = jobs[tile_job(s_tile0, njobs, t)];
        tile_fetch(smem_f, geom_of(J, t), grid_of(J), batch_rows(J.H) + 2 * hk, set, bar);
    };
    int t = running(blockIdx.x), n = 0;
    fetch(t, 0);
    for (int nt; t < ntiles; t = nt, n++) {
        const int j = tile_job(s_tile0, njobs, t);
        nt = running(t + (int)gridDim.x);
        const TileJob &J = jobs[j];
        if (!tile_run<false, NARROW>(smem_f, geom_of(J, t), grid_of(J), hk, s_kr[j], n, bar, J.w32, mx,
                                     [&]() { fetch(nt, (n + 1) & 1); })) {
            if (threadIdx.x == 0) atomicCAS(&J.ctl->error, 0, PCD_TIMEOUT);
            break;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (s_last) {
        __threadfence();
        for (int j = threadIdx.x; j < njobs; j += kTThreads) {
            if (s_kr[j] < 1) continue;
            volatile Ctl *c = jobs[j].ctl;
            c->stream_out = par ? 0 : 1;
            const int sw = c->sweeps + s_kr[j];
            c->sweeps = sw;
            if (sw >= jobs[j].max_iter) c->halt = 1;
        }
        if (threadIdx.x == 0) *counter = 0u;
        __threadfence();
    }
}

const void *tile_kernel(bool track, bool narrow)
{
    if (narrow) return track ? (const void *)k_tile_pass<true, true> : (const void *)k_tile_pass<false, true>;
    return track ? (const void *)k_tile_pass<true, false> : (const void *)k_tile_pass<false, false>;
}

const void *batch_kernel(bool narrow)
{
    return narrow ? (const void *)k_tile_batch<true> : (const void *)k_tile_batch<false>;
}

}  // namespace

int tile_plan(int dev, int W, int H, int ld, int depth, TilePlan *plan)
{
    if (W < 8 || H < 1 || W % 8 != 0 || ld % 4 != 0) return PCD_BAD_ARG;
    if (depth != 0 && depth != 2 && depth != 4) return PCD_BAD_ARG;
    TilePlan p;
    p.K = depth ? depth : kTilePassSweeps;
    p.ncol = ceil_div(W / 8, kTCL - 2);
    p.nrow = ceil_div(H, kTRows - 4 * p.K);
    p.smem = tile_smem();
    int sms = 0;
    PCD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    int bps = 1;
    for (bool track : {false, true}) {
        const void *fn = tile_kernel(track, W == 8);
        int b = 0;
        PCD_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p.smem));
        PCD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, fn, kTThreads, p.smem));
        bps = std::min(bps, b);
    }
    if (bps < 1) return PCD_BAD_ARG;
    // as many tile rows as the last round of CTAs has room for: shorter tiles
    // instead of a round that is nearly empty
    const long most = (long)sms * bps, rounds = ((long)p.ncol * p.nrow + most - 1) / most;
    p.nrow = (int)std::max<long>(p.nrow, std::min<long>(rounds * most / p.ncol, ceil_div(H, 16)));
    p.rows = 2 * ceil_div(H, 2L * p.nrow);
    p.nrow = ceil_div(H, p.rows);
    p.grid = (int)std::min<long>((long)p.ncol * p.nrow, most);
    *plan = p;
    return PCD_OK;
}

int tile_maps(const float *ea, const float *eb, const float *r32, int W, int H, int rows, TileMaps *m)
{
    const auto fn = tensor_map_encoder();
    if (!fn) {
        set_error("tile SOR: cuTensorMapEncodeTiled is not available");
        return PCD_DEVICE_ERROR;
    }
    const cuuint64_t KQ = (cuuint64_t)W / 8;
    const cuuint64_t dims[3] = {4 * KQ, 2, (cuuint64_t)H}, strides[2] = {16 * KQ, 32 * KQ};
    const cuuint32_t box[3] = {4 * kTCL, 1, (cuuint32_t)rows}, estr[3] = {1, 1, 1};
    const float *src[3] = {ea, eb, r32};
    CUtensorMap *map[3] = {&m->ea, &m->eb, &m->r32};
    for (int i = 0; i < 3; i++) {
        const CUresult r = fn(map[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float *>(src[i]), dims, strides,
                              box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) {
            set_error("tile SOR: cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")");
            return PCD_DEVICE_ERROR;
        }
    }
    return PCD_OK;
}

int launch_tile(const TilePlan &p, const CUtensorMap &ein, float *eout, const CUtensorMap &r32, Ctl *ctl,
                const SolveArgs &a, int nsw, int out_idx, bool track, bool zero, cudaStream_t s)
{
    if (nsw < 1 || nsw > p.K) {
        set_error("tile SOR: more sweeps than the plan's halo holds");
        return PCD_BAD_ARG;
    }
    using Fn = void (*)(CUtensorMap, float *, CUtensorMap, Ctl *, SolveArgs, int, int, int, int, int, int, int);
    const Fn fn = reinterpret_cast<Fn>(const_cast<void *>(tile_kernel(track, a.W == 8)));
    fn<<<p.grid, kTThreads, p.smem, s>>>(ein, eout, r32, ctl, a, p.ncol, p.nrow, p.rows, 2 * p.K, nsw, out_idx, zero ? 1 : 0);
    return PCD_OK;
}

int tile_job_setup(TileJob *job)
{
    job->ncol = ceil_div(job->W / 8, kTCL - 2);
    job->nrow = ceil_div(job->H, batch_rows(job->H));
    return tile_maps(job->ea, job->eb, job->r32, job->W, job->H, batch_rows(job->H) + 4 * kTilePassSweeps, &job->maps);
}

int tile_batch_config(int dev, int njobs, bool narrow, size_t *smem, int *grid)
{
    if (njobs < 1 || njobs > kTileBatchJobsMax) {
        set_error("batched tile pass: 1 to " + std::to_string(kTileBatchJobsMax) + " grids");
        return PCD_BAD_ARG;
    }
    const void *fn = batch_kernel(narrow);
    const size_t per_job = 2 * sizeof(int);
    const size_t most = tile_smem() + kTileBatchJobsMax * per_job, bytes = tile_smem() + (size_t)njobs * per_job;
    int sms = 0, bps = 0;
    PCD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    PCD_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
    PCD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, fn, kTThreads, bytes));
    if (bps < 1) {
        set_error("batched tile pass: the kernel does not fit on an SM");
        return PCD_BAD_ARG;
    }
    *smem = bytes;
    *grid = sms * bps;
    return PCD_OK;
}

int launch_tile_batch(const TileJob *d_jobs, int njobs, int ntiles, int nsw, int par, bool zero, bool narrow, int grid,
                      size_t smem, unsigned *counter, cudaStream_t s)
{
    if (njobs < 1 || njobs > kTileBatchJobsMax || ntiles < 1 || nsw < 1 || nsw > kTilePassSweeps) {
        set_error("batched tile pass: bad arguments");
        return PCD_BAD_ARG;
    }
    using Fn = void (*)(const TileJob *, int, int, int, int, int, unsigned *);
    const Fn fn = reinterpret_cast<Fn>(const_cast<void *>(batch_kernel(narrow)));
    fn<<<std::min(grid, ntiles), kTThreads, smem, s>>>(d_jobs, njobs, ntiles, nsw, par, zero ? 1 : 0, counter);
    return PCD_OK;
}

}  // namespace pcd
