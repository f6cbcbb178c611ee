// sor_passes.cuh -- FP32 red-black SOR passes over grids in HBM (internal).
#pragma once

#include <cuda.h>

#include "solver.cuh"

namespace pcd {

// Register-resident tile passes for grids in HBM (FP32 correction sweeps, the
// correction and minus its right-hand side in the layout of sor_quads.cuh,
// ping-pong buffers): K sweeps per pass, ncol x nrow tiles of `rows` written rows
// on `grid` persistent CTAs.
constexpr int kTilePassSweeps = 4;
struct TilePlan {
    int K = 0;
    int ncol = 0, nrow = 0, rows = 0, grid = 0;
    size_t smem = 0;
};

// A grid's arrays as the passes' TMA copies see them, boxes of one plane (the
// cells in even or in odd columns): the two corrections and minus their right-hand
// side as read, a tile's rows and lane columns with their halo, and the
// corrections as written, without it (lane columns: KQ / ncol, and one more).
struct TileMaps {
    CUtensorMap in[2], out[2][2], r32;
};
// Tiles of `rows` written rows and `halo` more on each side, ncol tile columns.
int tile_maps(float *ea, float *eb, const float *r32, int W, int H, int ncol, int rows, int halo, TileMaps *m);

// One grid of a batched tile pass (4 sweeps at most).
struct TileJob {
    TileMaps maps;
    float *ea, *eb;      // FP32 correction buffers (ping-pong)
    const float *r32;    // minus the FP32 right-hand side
    Ctl *ctl;            // the grid's control block
    int W, H;            // W a multiple of 8
    int ncol, nrow;      // tiles
    int tile0;           // first global tile index of the grid
    int max_iter;
    float w32[5];        // omega / cnt
};

// The batched form's tiles of a job's grid (W, H and the buffers are set):
// ncol, nrow and maps.
int tile_job_setup(TileJob *job);
// Most grids in one batched pass (two words a grid sit in shared memory).
constexpr int kTileBatchJobsMax = 1024;
// Dynamic shared memory of the batched pass for njobs grids (narrow: some of
// them 8 cells wide) and its persistent grid.
int tile_batch_config(int dev, int njobs, bool narrow, size_t *smem, int *grid);
// `sweeps` sweeps (fewer at a grid's sweep cap) in passes of four over ntiles
// tiles of njobs grids (d_jobs on the device, tile0 ascending), the corrections
// starting from 0 in ea.  Cooperative.  sync (two words), done (one a tile):
// zero before a solve's first launch; limit: polls before a wait gives up;
// withhold: tile 0 is never reported done.
int launch_tile_batch(const TileJob *d_jobs, int njobs, int ntiles, int sweeps, bool narrow, int grid, size_t smem,
                      unsigned *sync, unsigned *done, long long limit, int withhold, cudaStream_t s);

// The plan for a W x H grid (W >= 8); depth = sweeps per pass (2 or 4; 0: 4).
// PCD_BAD_ARG when no form applies.
int tile_plan(int dev, int W, int H, int depth, TilePlan *plan);
// `sweeps` sweeps (fewer at the sweep cap), nsw <= K in a pass, of a correction that
// starts from 0; the result ping-pongs between the maps' buffers
// (Ctl::stream_out).  Cooperative.  The max-update stop is tested for every pass
// (each; a second launch stops where it was met) or for the last one (gmax: a word
// a pass, zero between launches).  done: a word a tile, zero before a solve's first launch;
// limit: polls before a wait gives up; withhold: tile 0 is never reported done.
int launch_tile(const TilePlan &p, const TileMaps &maps, Ctl *ctl, unsigned *done, unsigned *gmax, const SolveArgs &a,
                int nsw, int sweeps, bool each, long long limit, int withhold, cudaStream_t s);

}  // namespace pcd
