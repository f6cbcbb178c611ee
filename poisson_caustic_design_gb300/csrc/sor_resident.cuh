// sor_resident.cuh -- FP32 red-black SOR on tiles that stay on the chip for a
// whole cycle of sweeps (internal).
#pragma once

#include "solver.cuh"

namespace pcd {

constexpr int kResidentChecksMax = 512;  // tracked sweeps of one launch
constexpr int kResidentCtasMax = 256;

struct ResidentArgs {
    int W, H;
    int KQ;              // lane columns of the grid (8 cells each)
    int TX, TY;          // tile columns x tile rows = CTAs
    int NG, R;           // row groups of a CTA, most rows of any tile (halo included)
    float *e;            // FP32 correction, out (in the layout of sor_quads.cuh, as r32)
    const float *r32;    // minus the FP32 right-hand side
    Ctl *ctl;
    void *xb;            // exchange words: [2 parities][2 colours][H][KQ] x 32 bytes
    unsigned long long *part;  // residual partials: [2][CTAs] words
    unsigned *gmax;      // tracked maxima (zero between launches)
    unsigned *bar;       // grid barrier counter (zero between launches)
    int nsw;             // sweeps of this launch at most
    int max_iter;
    int cycle;           // 1: end on the residual estimate; 0: run nsw sweeps
    int check_every;     // cycle: sweeps between estimates,
    int dep, lag;        //   each on a multiple of dep; the cycle ends lag sweeps after it
    int gran;            // max-update stop: tracked every gran sweeps; 0: not tracked
    double tol, drop;
    float w32[5];
    long long spin_limit;
    int withhold;        // failure test: CTA 0 never publishes
};

// One launch shape: sweeps per halo exchange (K), rows of a lane (L), lanes of
// a tile row (CL), tiles, warps and row groups of a CTA.
struct ResidentPlan {
    int K = 0, L = 0, CL = 0;
    int TX = 0, TY = 0, NW = 0, NG = 0, R = 0, KQ = 0;
    size_t smem = 0;
    size_t xb_bytes = 0;
};

// PCD_BAD_ARG when the grid does not fit on the chip.
int resident_plan(int dev, int W, int H, ResidentPlan *plan);
int launch_resident(ResidentArgs &a, const ResidentPlan &p, cudaStream_t s);

}  // namespace pcd
