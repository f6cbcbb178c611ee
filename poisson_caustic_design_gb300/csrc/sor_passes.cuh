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

// A grid's arrays as the passes' bulk copies see them: boxes of one plane (the
// cells in even or in odd columns) of a tile's rows x lane columns.
struct TileMaps {
    CUtensorMap ea, eb, r32;
};
// rows: of a tile, halo included.
int tile_maps(const float *ea, const float *eb, const float *r32, int W, int H, int rows, TileMaps *m);

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
// One batched pass of nsw <= 4 sweeps over ntiles tiles of njobs grids
// (d_jobs on the device, tile0 ascending); parity par reads ea (0) or eb, zero:
// the corrections start from 0.
// counter: a device word that is zero between passes.
int launch_tile_batch(const TileJob *d_jobs, int njobs, int ntiles, int nsw, int par, bool zero, bool narrow, int grid,
                      size_t smem, unsigned *counter, cudaStream_t s);

// The plan for a W x H grid with leading dimension ld (W a multiple of 8, ld
// of 4); depth = sweeps per pass (2 or 4; 0: 4).  PCD_BAD_ARG when no form
// applies.
int tile_plan(int dev, int W, int H, int ld, int depth, TilePlan *plan);
// One pass of nsw <= K sweeps from ein into eout (fewer at the sweep cap);
// track: the pass reports the largest |update| of its last sweep; zero: the
// correction starts at 0 and ein is not read.
int launch_tile(const TilePlan &p, const CUtensorMap &ein, float *eout, const CUtensorMap &r32, Ctl *ctl,
                const SolveArgs &a, int nsw, int out_idx, bool track, bool zero, cudaStream_t s);

}  // namespace pcd
