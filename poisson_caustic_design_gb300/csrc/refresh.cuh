// refresh.cuh -- the FP64 passes of a solve: its start and the refresh of a
// mixed-precision solve's residual (internal).
#pragma once

#include "solver.cuh"

namespace pcd {

// One grid of a refresh launch: blocks [blk0, blk0 + nblk) work on it.
struct RefreshJob {
    const double *b;
    double *phi, *phi2;      // the potential alternates between the two (ctl->phi_side)
    const float *e0, *e1;    // the correction: e1 when ctl->stream_out is set
    float *r32;              // minus the right-hand side (both in the layout of sor_quads.cuh)
    Ctl *ctl;
    const int *error;        // of the solve: the control block's, or the one that a batch shares
    double *partials;        // 3 per block
    int W, H, ld;
    int blk0, nblk;
    int rows;                // rows of a strip piece
    // a single solve's launches leave their control block here (host memory), and
    // one behind the solve's last brings the potential back into phi
    Ctl *report;
};

// Blocks of a W x H grid's refresh (at most cap) on sms SMs, a batch's grid on its
// share of them, and the rows of a piece.  ld < kRefreshLdMax.
constexpr int kRefreshLdMax = 1 << 26;
int refresh_shape(int W, int H, int ld, int cap, double sms, int *rows);
// For every job whose solve is not done and has no error: phi += e in FP64, r = b -
// L phi, -r in FP32 to r32, the norms, and (tol >= 0) the relative-residual stop
// test; a solve that has halted is then done.  jobs: on the device, or nullptr for
// the single job `one`.
int launch_refresh(const RefreshJob *jobs, const RefreshJob &one, int njobs, int blocks, double tol, cudaStream_t s);
// The same for the starts of a batch: e is 0 (zero: so is phi), the norms
// include ||b||, and phi stays where it is.
int launch_first_refresh(const RefreshJob *jobs, int njobs, int blocks, double tol, bool zero, cudaStream_t s);
// A batch's potentials back into phi.
int launch_phi_settle(const RefreshJob *jobs, int njobs, cudaStream_t s);

// The start of a solve: the neighbour-validity mask and the number of NaN
// cells of b; zero: phi = 0; r = b - L phi in FP64 over the valid cells with
// ||b||, ||r||, max |r| and (test) the relative-residual stop test, which
// leaves the solve done where it passes; r64 / r32 (may be nullptr) receive r,
// r32 row-major or (quads) negated and in the layout of sor_quads.cuh.
int launch_start(const double *b, double *phi, uint8_t *mask, double *r64, float *r32, Ctl *ctl, double *partials,
                 int max_partials, const SolveArgs &a, bool zero, bool quads, bool test, cudaStream_t s);

}  // namespace pcd
