// sor_blocks64.cuh -- persistent FP64 red-black SOR over 2-D blocks (internal).
#pragma once

#include "solver.cuh"

namespace pcd {

struct Blocks64Args {
    int W, H, ld;
    int TY, TX, G;        // block rows x block columns = CTAs
    int K, RTmax;         // sweeps per exchange (halo 2K cells), most region rows
    const double *b;
    double *phi;
    void *xb;             // exchange words: [2 parities][H][ceil(W/2)] x 32 bytes, zeroed
    void *part;           // check partials: [2][G] x 32 bytes, zeroed
    Ctl *ctl;
    int stop, max_iter, check_every;
    double tol, omega;
    double w64[5];
    long long spin_limit;
    int withhold;         // failure test: CTA 0 never publishes
};

struct Blocks64Plan {
    int TY = 0, TX = 0, K = 0, RTmax = 0;
    size_t smem = 0, xb_bytes = 0;
};
// K > 0: that many sweeps per exchange; 0: chosen by the expected time.
// PCD_BAD_ARG when no layout fits.
int blocks64_plan(int dev, int W, int H, int K, Blocks64Plan *plan);
int launch_blocks64(Blocks64Args &a, const Blocks64Plan &p, cudaStream_t s);

}  // namespace pcd
