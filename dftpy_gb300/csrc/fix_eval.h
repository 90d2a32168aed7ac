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

// Kernel classes of these evaluations, and who times them (ofdft_eval_profile; owner null: nobody):
// a launch, or a few of one class, between begin and end, with the bytes that it has to move
enum Part { PRE, POST, SUMS, FFT, NODES, AXIS1, INTERP, HATS, POT2 };
struct Timing {
    void* owner = nullptr;
    int (*begin)(void* owner, Part part, double bytes, cudaStream_t st) = nullptr;
    void (*end)(void* owner, int at, cudaStream_t st) = nullptr;
    template <class F>
    void operator()(Part part, double bytes, cudaStream_t st, F&& f) const {
        const int at = owner ? begin(owner, part, bytes, st) : -1;
        f();
        OFDFT_LAUNCH_CHECK();
        if (owner) end(owner, at, st);
    }
};

struct LocalArgs {
    Timing time;
    const double* rho;
    const double* vloc;  // or null
    double* V;           // or null: energies only
    int tf, vw, wt, lwt, xc, h;
    double tf_x, vw_y;
    double alpha, beta;  // exponents of the nonlocal term
    double wt_x, wt_rho0;
    double* wtstate;  // [rho0, rebuild, 2 k_F, factor, built]
    double* wtK;      // kernel at the state's rho0 (Nc)
    double cTF_wt;
};

// The density-dependent kernel between the two halves of an evaluation (fix_lwt.cu)
struct LwtArgs {
    Timing time;
    const double* kf;
    const double* rA;
    const double2* rbG;  // FFT(rho^beta)
    // out: pot2, and pot1 and pot3 (kdd = 3) as sums of arrays (lwt_has)
    double *pot1[4], *pot2, *pot3[4];
    const double *tab_c, *tab_cd, *tab_x;  // kernel table, derivative table, knots
    int nint;
    double step, etamax, limit, limitd;
    const double *kn, *invk, *kup;  // nodes, reciprocals, nodes + 1e-18 (device)
    int m, kdd, hermite, max_batch;
    double kfclip;
};
// The arrays that make up pot1 and pot3: contributions of a point's lower and upper nodes
// (0, 2: kernel planes, 1, 3: derivative planes); linear interpolation has no derivative part
// in pot1 and no other in pot3
inline bool lwt_has(int pot, int part, bool hermite) { return hermite || (part & 1) == (pot == 3); }
int lwt_enqueue(ofdft_grid* g, Scratch& sc, const LwtArgs& r, cudaStream_t st);

// An evaluation in two halves: the pre-pass and the transforms of the local terms; the
// post-pass.  Sums go to d_results as the evaluator lays them out: [0] TF, [1] XC, [2] PP,
// [3] sum rho, [4] min k_F, [5] max k_F, [6] max rho (the last three with lwt, and copied to
// h_results when `copied` fires), [16] vW, [17] Hartree, [18] WT or LWT.  Both return the
// number of launches.
struct Fields {
    double *sq = nullptr, *rb = nullptr, *ra = nullptr, *kf = nullptr;
    double *vH = nullptr, *lap = nullptr, *nl1 = nullptr, *nl2 = nullptr;
    double2* rbG = nullptr;  // FFT(rho^beta), with lwt
};
struct LwtPost {
    const double *pot1[4] = {}, *pot2 = nullptr, *pot3[4] = {};
    double rhomax = 0, ld = 0, kfclip = 0;
};
int local_begin(ofdft_grid* g, Scratch& sc, const LocalArgs& a, Fields& f, cudaEvent_t copied, cudaStream_t st);
int local_finish(ofdft_grid* g, Scratch& sc, const LocalArgs& a, const Fields& f, const LwtPost& q, cudaStream_t st);

}  // namespace fix
}  // namespace ofdft
