// Float64 evaluation of the local terms and of the density-independent nonlocal
// term with integer-pipe transforms (fix_eval.cu).
#pragma once
#include "common.cuh"

namespace ofdft {
namespace fix {

struct Grid3;

// The transform plans of a float64 grid (built on first use, kept with the grid), or
// nullptr when an axis has a prime factor above 7 or is longer than the plans cover.
const Grid3* grid_plans(ofdft_grid* g);
void free_plans(ofdft_grid* g);

// R2C / C2R of nf fields (cuFFT's layouts, unnormalised); the C2R overwrites its input
void r2c(ofdft_grid* g, const double* const* in, double2* const* out, int nf, cudaStream_t st);
void c2r(ofdft_grid* g, double2* const* in, double* const* out, int nf, cudaStream_t st);

struct LocalArgs {
    const double* rho;
    const double* vloc;  // or null
    double* V;           // or null: energies only
    int tf, vw, wt, xc, h;
    double tf_x, vw_y;
    double wt_alpha, wt_beta, wt_x, wt_rho0;
    double* wtstate;  // [rho0, rebuild, 2 k_F, factor, built]
    double* wtK;      // kernel at the state's rho0 (Nc)
    double cTF_wt;
};

// Enqueues the evaluation; sums in d_results as the evaluator lays them out:
// [0] TF, [1] XC, [2] PP, [3] sum rho, [16] vW, [17] Hartree, [18] WT.  Returns the
// number of launches.
int local_enqueue(ofdft_grid* g, Scratch& sc, const LocalArgs& a, cudaStream_t st);

}  // namespace fix
}  // namespace ofdft
