// sor_cluster.cuh -- FP32 red-black SOR on one thread-block cluster (internal).
#pragma once

#include "solver.cuh"

namespace pcd {

constexpr int kClusterThreads = 1024;

struct ClusterArgs {
    int W, H, ld;
    int khp;             // shared-memory row stride of a colour plane (multiple of 4)
    float *e;            // FP32 correction (global, ld-strided), in/out
    const float *r32;    // FP32 right-hand side
    Ctl *ctl;            // reads bnorm / rnorm / sweeps, writes sweeps / halt
    int check_every;     // sweeps between FP32 residual estimates
    int cycle_cap;       // sweeps per cycle at most
    int max_iter;        // total sweep cap
    double tol;          // relative stop tolerance
    double drop;         // end the cycle when the estimate fell by this factor
    float w32[5];        // omega / cnt
    float one_minus_omega;
    int depth;           // sweeps between halo exchanges (1, 2 or 4; 0: one exchange per half sweep)
};

// How one grid runs on one cluster: C CTAs (16 or 8), dynamic shared memory,
// the shared-memory plane stride, the sweeps per halo exchange (0: one
// exchange per half sweep) and, for the register-resident form, the rows per
// warp and quads per lane (rr_l = 0: the shared-memory forms).
struct ClusterPlan {
    int C;
    size_t smem;
    int khp;
    int depth;
    int rr_l;
    int rr_nq;
};

// The plan for a W x H grid; PCD_BAD_ARG when the grid does not fit in one
// cluster.  max_depth caps the sweeps per exchange (0: the per-half-sweep
// exchange; the register-resident form needs at least 2).
int cluster_plan(int dev, int W, int H, int max_depth, ClusterPlan *plan);
int launch_cluster(ClusterArgs &a, const ClusterPlan &p, cudaStream_t s);

}  // namespace pcd
