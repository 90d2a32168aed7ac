// Ewald ion-ion energy and forces (src/dftpy/ewald.py:197-864).
//   eta        Get_Best_eta (:256-278), on the host
//   real part  erfc(sqrt(eta) r)/r over all images within Rcut (Energy_real
//              :281-325, Forces_real :541-577), from a cell list
//   reciprocal smooth PME (Energy_rec_PME :786-807, Forces_rec_PME :810-864)
//              or exact structure factors (Energy_rec :449-466, Forces_rec :580-607)
//   correction Energy_corr (:468-482), on the host
//   stress     Stress_real (:609-662) with the real-space sum; Stress_rec_PME
//              (:915-968) or Stress_rec (:719-763) over the mask, G = 0 term
#include "common.cuh"
#include "fix_eval.h"
#include "host_math.h"
#include "pme.cuh"

#include <algorithm>
#include <cstring>

using namespace ofdft;

namespace ofdft {
void frac_coords(const double* lattice, int nat, const double* pos, std::vector<double>& frac);
void lattice_inverse(const double* a, double* inv);
void bspline_tables(const ofdft_grid* g, int order, std::vector<double>& re, std::vector<double>& im);
}  // namespace ofdft

namespace {

struct CellList {
    int nc[3];
    int K[3];
    const int* start;   // nc0*nc1*nc2 + 1
    const int* atoms;   // atom indices sorted by cell
    const int* cellof;  // cell of each atom
};

// One warp per atom over the atoms of the (2K+1)^3 neighbour cells (unwrapped, so each
// periodic image of each atom is visited exactly once), 32 candidates at a time: every lane
// computes one candidate's terms, then ten lanes add one component each, in the order of
// the candidates, so the sums are those of a serial loop (the optimisers' line searches
// see the energy's last bits).  One thread per atom took 143 us, a serial chain of float64
// functions.  Per atom: the energy sum, then the six sums of Stress_real (:645-654),
// q_i q_j (2 sqrt(eta/pi) exp(-eta d^2) + erfc(sqrt(eta) d)/d) R_a R_b / d^2, to sums[7 i].
constexpr int kRealWarps = 4;
__global__ void __launch_bounds__(32 * kRealWarps)
    k_ewald_real(const double* __restrict__ pos, const double* __restrict__ q, int nat, const double* __restrict__ lat,
                 CellList cl, double Rcut, double eta, double* F, double* __restrict__ sums) {
    __shared__ double term[kRealWarps][32][10];
    __shared__ int first[kRealWarps][32];  // candidates before each cell of the batch
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int i = blockIdx.x * kRealWarps + warp;
    if (i >= nat) return;
    const double es = sqrt(eta);
    const double rtol = 0.001;
    const double xi = pos[3 * i], yi = pos[3 * i + 1], zi = pos[3 * i + 2];
    const int c = cl.cellof[i];
    const int c0 = c / (cl.nc[1] * cl.nc[2]), c1 = (c / cl.nc[2]) % cl.nc[1], c2 = c % cl.nc[2];
    const double sp2 = 2.0 * es / sqrt(M_PI);
    const int m1 = 2 * cl.K[1] + 1, m2 = 2 * cl.K[2] + 1, cells = (2 * cl.K[0] + 1) * m1 * m2;
    double s = 0.0;  // component `lane` < 10: energy, force, stress
    auto unwrapped = [&](int t, int (&u)[3]) {
        u[0] = c0 + t / (m1 * m2) - cl.K[0];
        u[1] = c1 + (t / m2) % m1 - cl.K[1];
        u[2] = c2 + t % m2 - cl.K[2];
    };
    auto cell_of = [&](const int (&u)[3]) {
        return (pmod(u[0], cl.nc[0]) * cl.nc[1] + pmod(u[1], cl.nc[1])) * cl.nc[2] + pmod(u[2], cl.nc[2]);
    };
    for (int t0 = 0; t0 < cells; t0 += 32) {
        // the batch's cells, one per lane, and where their atoms start in its candidates
        int u[3], count = 0;
        if (t0 + lane < cells) {
            unwrapped(t0 + lane, u);
            const int cell = cell_of(u);
            count = cl.start[cell + 1] - cl.start[cell];
        }
        int upto = count;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += x;
        }
        __syncwarp();
        first[warp][lane] = upto - count;
        __syncwarp();
        const int total = __shfl_sync(0xffffffffu, upto, 31);
        for (int h0 = 0; h0 < total; h0 += 32) {
            const int h = h0 + lane;
            bool in = false;
            if (h < total) {
                int lo = 0, hi = 32;  // the last cell that starts at or before h (empty ones share its start)
                while (hi - lo > 1) {
                    const int mid = (lo + hi) >> 1;
                    if (first[warp][mid] <= h) lo = mid;
                    else hi = mid;
                }
                unwrapped(t0 + lo, u);
                const int cell = cell_of(u);
                const int j = cl.atoms[cl.start[cell] + h - first[warp][lo]];
                const double n0 = floor((double)u[0] / cl.nc[0]), n1 = floor((double)u[1] / cl.nc[1]),
                             n2 = floor((double)u[2] / cl.nc[2]);
                const double tx = n0 * lat[0] + n1 * lat[3] + n2 * lat[6];
                const double ty = n0 * lat[1] + n1 * lat[4] + n2 * lat[7];
                const double tz = n0 * lat[2] + n1 * lat[5] + n2 * lat[8];
                const double dx = xi - (pos[3 * j] + tx), dy = yi - (pos[3 * j + 1] + ty),
                             dz = zi - (pos[3 * j + 2] + tz);
                const double d = sqrt(dx * dx + dy * dy + dz * dz);
                in = d < Rcut && d > rtol;
                if (in) {
                    const double x = es * d;
                    const double ec = erfc(x);
                    double* o = term[warp][lane];
                    o[0] = q[j] * ec / d;
                    const double w = q[j] * (ec / (x * x * x) + 2.0 / sqrt(M_PI) * exp(-x * x) / (x * x));
                    o[1] = dx * w;
                    o[2] = dy * w;
                    o[3] = dz * w;
                    const double ws = q[j] * (sp2 * exp(-eta * d * d) + ec / d) / (d * d);
                    o[4] = ws * dx * dx;
                    o[5] = ws * dx * dy;
                    o[6] = ws * dx * dz;
                    o[7] = ws * dy * dy;
                    o[8] = ws * dy * dz;
                    o[9] = ws * dz * dz;
                }
            }
            unsigned hits = __ballot_sync(0xffffffffu, in);
            __syncwarp();
            if (lane < 10)
                for (; hits; hits &= hits - 1) s += term[warp][__ffs(hits) - 1][lane];
            __syncwarp();
        }
    }
    if (lane == 0) sums[7 * i] = q[i] * s;
    else if (lane < 4) F[3 * i + lane - 1] = q[i] * s * (es * es * es);
    else if (lane < 10) sums[7 * i + lane - 3] = q[i] * s;
}

// block sums of the atoms' seven values, one thread per atom
__global__ void __launch_bounds__(RED_THREADS) k_ewald_real_sum(const double* __restrict__ sums, int nat,
                                                                double* partials) {
    double acc[7] = {0, 0, 0, 0, 0, 0, 0};
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nat)
        for (int k = 0; k < 7; ++k) acc[k] = sums[7 * i + k];
    block_sum_store<7>(acc, partials);
}

// PME reciprocal energy and (conv) the force convolution's input, over QG in place:
// E = 4 pi/V sum_mask |Q(G) B(G)|^2 exp(-G^2/4 eta)/G^2 (raw FFT, dV factors cancel);
// X = Q(G) |B(G)|^2 exp(-G^2/4 eta)/G^2 / N.  The factors of the energy's terms go to
// terms (zero outside the mask) and are summed by k_ewald_rec_sum, whose order of the
// points does not depend on how this pass walks the rows.
template <typename T>
__global__ void __launch_bounds__(32 * kRowWarps)
    k_ewald_rec_pme(typename Cplx<T>::type* __restrict__ QG, bool conv, const double* bre, const double* bim, Geo geo,
                    double eta, double2* __restrict__ terms) {
    const int rows = geo.n0 * geo.n1;
    const double invN = 1.0 / (double)geo.N;
    for (int row = blockIdx.x * kRowWarps + (threadIdx.x >> 5); row < rows; row += gridDim.x * kRowWarps) {
        const HalfRow r = half_row(geo, row, bre, bim);
        for (int k = threadIdx.x & 31; k < geo.n2h; k += 32) {
            const long long i = (long long)row * geo.n2h + k;
            const double gg = row_gsq(geo, r, k);
            double br, bi;
            row_barray(geo, r, bre, bim, k, br, bi);
            const double qr = (double)QG[i].x, qi = (double)QG[i].y;
            const double sr = qr * br - qi * bi, si = qr * bi + qi * br;
            const double inv = (i == 0) ? 0.0 : 1.0 / gg;
            const double w = exp(-gg / (4.0 * eta)) * inv;
            terms[i] = half_mask(geo, i) ? make_double2(sr * sr + si * si, w) : make_double2(0.0, 0.0);
            if (conv) {
                const double f = (br * br + bi * bi) * w * invN;
                QG[i].x = (T)(qr * f);
                QG[i].y = (T)(qi * f);
            }
        }
    }
}

__global__ void __launch_bounds__(RED_THREADS) k_ewald_rec_sum(const double2* __restrict__ terms, long long n,
                                                               double* partials) {
    double acc[1] = {0.0};
    const long long stride = (long long)gridDim.x * blockDim.x;
#pragma unroll 4
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += stride) {
        const double2 t = terms[i];
        acc[0] = fma(t.x, t.y, acc[0]);
    }
    block_sum_store<1>(acc, partials);
}

// exact structure factor S(G) = sum_a q_a exp(-i G.R_a) and the energy sum
template <typename T>
__global__ void __launch_bounds__(RED_THREADS) k_ewald_rec_exact(const double* __restrict__ pos,
                                                                 const double* __restrict__ q, int nat, Geo geo,
                                                                 double eta, double* S, double* partials) {
    double acc[1] = {0.0};
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < geo.Nc; i += stride) {
        double gx, gy, gz, gg;
        gvec(geo, i, gx, gy, gz, gg);
        double sr = 0.0, si = 0.0;
        for (int a = 0; a < nat; ++a) {
            double ph = gx * pos[3 * a] + gy * pos[3 * a + 1] + gz * pos[3 * a + 2];
            double sn, cs;
            sincos(ph, &sn, &cs);
            sr += q[a] * cs;
            si -= q[a] * sn;
        }
        S[2 * i] = sr;
        S[2 * i + 1] = si;
        double inv = (i == 0) ? 0.0 : 1.0 / gg;
        if (half_mask(geo, i)) acc[0] += (sr * sr + si * si) * exp(-gg / (4.0 * eta)) * inv;
    }
    block_sum_store<1>(acc, partials);
}

// Reciprocal stress sums over the mask (Stress_rec_PME :937-950, Stress_rec
// :733-751): |S(G)|^2 exp(-G^2/4 eta)/G^2 (2 g_i g_j/G^2 (1 + G^2/4 eta) - delta_ij)
// with S = FFT(Q) B (PME, raw transform) or the exact structure factor.
template <typename T>
__global__ void __launch_bounds__(RED_THREADS) k_ewald_stress_rec(const typename Cplx<T>::type* __restrict__ QG,
                                                                  const double* __restrict__ S, const double* bre,
                                                                  const double* bim, Geo geo, double eta,
                                                                  double* partials) {
    double acc[6] = {0, 0, 0, 0, 0, 0};
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < geo.Nc; i += stride) {
        if (!half_mask(geo, i)) continue;
        double gx, gy, gz, gg;
        gvec(geo, i, gx, gy, gz, gg);
        double sr, si;
        if (QG) {
            double br, bi;
            barray(bre, bim, geo, i, br, bi);
            const double qr = (double)QG[i].x, qi = (double)QG[i].y;
            sr = qr * br - qi * bi;
            si = qr * bi + qi * br;
        } else {
            sr = S[2 * i];
            si = S[2 * i + 1];
        }
        const double inv = (i == 0) ? 0.0 : 1.0 / gg;
        const double w = (sr * sr + si * si) * exp(-gg / (4.0 * eta)) * inv;
        const double f = 2.0 * inv * (1.0 + gg / (4.0 * eta));
        const double g[3] = {gx, gy, gz};
        int k = 0;
        for (int a = 0; a < 3; ++a)
            for (int b = a; b < 3; ++b, ++k) acc[k] += w * (g[a] * g[b] * f - (a == b ? 1.0 : 0.0));
    }
    block_sum_store<6>(acc, partials);
}

constexpr int kChunk = 8;

// exact reciprocal forces for a chunk of atoms:
// F_a = 8 pi/V sum_mask G (Re s_a Im S - Im s_a Re S) exp(-G^2/4eta)/G^2, s_a = q_a e^{-iG.R_a}
__global__ void __launch_bounds__(RED_THREADS) k_ewald_force_exact(const double* __restrict__ pos,
                                                                   const double* __restrict__ q, const double* S,
                                                                   int a0, int na, Geo geo, double eta,
                                                                   double* partials) {
    double acc[3 * kChunk];
    for (int t = 0; t < 3 * kChunk; ++t) acc[t] = 0.0;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < geo.Nc; i += stride) {
        if (!half_mask(geo, i)) continue;
        double gx, gy, gz, gg;
        gvec(geo, i, gx, gy, gz, gg);
        double inv = (i == 0) ? 0.0 : 1.0 / gg;
        double w = exp(-gg / (4.0 * eta)) * inv;
        double Sr = S[2 * i], Si = S[2 * i + 1];
        for (int t = 0; t < na; ++t) {
            const int a = a0 + t;
            double ph = gx * pos[3 * a] + gy * pos[3 * a + 1] + gz * pos[3 * a + 2];
            double sn, cs;
            sincos(ph, &sn, &cs);
            double sr = q[a] * cs, si = -q[a] * sn;
            double den = (sr * Si - si * Sr) * w;
            acc[3 * t] += gx * den;
            acc[3 * t + 1] += gy * den;
            acc[3 * t + 2] += gz * den;
        }
    }
    block_sum_store<3 * kChunk>(acc, partials);
}

double best_eta(double precision, double gmax, const std::vector<double>& q) {
    double q2 = 0.0;
    for (double x : q) q2 += x * x;
    const double nat = (double)q.size();
    double eta = 1.6;
    for (int it = 0; it < 100000; ++it) {
        double up = 4.0 * M_PI * nat * q2 * std::sqrt(eta / M_PI) * std::erfc(gmax / 2.0 * std::sqrt(1.0 / eta));
        if (up < precision) return eta;
        eta = eta - 0.01;
        if (eta <= 0.0) break;
    }
    set_error("Ewald: no eta satisfies precision %g", precision);
    throw Error{OFDFT_EINVAL};
}

template <typename T>
void ewald_t(ofdft_grid* g, int nat, const double* pos, const double* charges, double precision, int pme, int order,
             double* out_energy, double* forces, double* out_eta, double* stress, cudaStream_t st) {
    using C = typename Cplx<T>::type;
    std::vector<double> q(charges, charges + nat);
    // gmax = sqrt(2 ecut), ecut from the grid spacing (grid.py:363-366, :722-723)
    double lengths[3], sp[3];
    for (int d = 0; d < 3; ++d) {
        const double* a = g->lattice + 3 * d;
        lengths[d] = std::sqrt(a[0] * a[0] + a[1] * a[1] + a[2] * a[2]);
        sp[d] = 0.5 * (lengths[d] / g->nr[d] + lengths[d] / (g->nr[d] - 1));
    }
    double spmax = std::max(sp[0], std::max(sp[1], sp[2]));
    double ecut = M_PI * M_PI / (2 * spmax * spmax);
    const double gmax = std::sqrt(2.0 * ecut);
    const double eta = best_eta(precision, gmax, q);
    if (out_eta) *out_eta = eta;
    const double Rcut = erfcinv_host(precision / 3.0) / std::sqrt(eta);

    // ---- correction (ewald.py:468-482)
    double q2 = 0.0, qs = 0.0;
    for (double x : q) {
        q2 += x * x;
        qs += x;
    }
    const double e_corr = -std::sqrt(eta / M_PI) * q2 - 4.0 * M_PI * (1.0 / (4.0 * eta * g->volume) / 2.0) * qs * qs;

    // ---- real space on a cell list
    std::vector<double> frac;
    frac_coords(g->lattice, nat, pos, frac);
    std::vector<double> wpos(3 * (size_t)nat);
    for (int a = 0; a < nat; ++a)
        for (int k = 0; k < 3; ++k)
            wpos[3 * a + k] = frac[3 * a] * g->lattice[k] + frac[3 * a + 1] * g->lattice[3 + k] +
                              frac[3 * a + 2] * g->lattice[6 + k];
    // perpendicular widths w_d = V / |a_e x a_f|
    const double* L = g->lattice;
    auto cross_norm = [&](int e, int f) {
        const double* u = L + 3 * e;
        const double* v = L + 3 * f;
        double cx = u[1] * v[2] - u[2] * v[1], cy = u[2] * v[0] - u[0] * v[2], cz = u[0] * v[1] - u[1] * v[0];
        return std::sqrt(cx * cx + cy * cy + cz * cz);
    };
    double wd[3] = {g->volume / cross_norm(1, 2), g->volume / cross_norm(0, 2), g->volume / cross_norm(0, 1)};
    CellList cl;
    for (int d = 0; d < 3; ++d) {
        cl.nc[d] = std::max(1, std::min(64, (int)std::floor(wd[d] / Rcut)));
        cl.K[d] = (int)std::ceil(Rcut * cl.nc[d] / wd[d]);
    }
    const int ncell = cl.nc[0] * cl.nc[1] * cl.nc[2];
    std::vector<int> cellof(nat), start(ncell + 1, 0), order_atoms(nat);
    for (int a = 0; a < nat; ++a) {
        int c[3];
        for (int d = 0; d < 3; ++d) c[d] = std::min(cl.nc[d] - 1, (int)(frac[3 * a + d] * cl.nc[d]));
        cellof[a] = (c[0] * cl.nc[1] + c[1]) * cl.nc[2] + c[2];
        start[cellof[a] + 1]++;
    }
    for (int c = 0; c < ncell; ++c) start[c + 1] += start[c];
    {
        std::vector<int> fill(start.begin(), start.end() - 1);
        for (int a = 0; a < nat; ++a) order_atoms[fill[cellof[a]]++] = a;
    }
    // Device buffers live in the grid's scratch; what the host prepares goes up in one copy.
    // Meshes above kKeep bytes are the call's own and are freed with it, as large grids need the
    // memory for node planes.  Allocating and freeing two of 135 MB (256^3; kept) takes 0.3 ms of
    // a 6.5 ms ion step, two of 540 MB 1.0 ms.
    constexpr size_t kKeep = (size_t)320 << 20;
    Scratch& sc = g->scratch;
    Scratch own;
    const size_t n = (size_t)nat;
    double cinv[9];
    lattice_inverse(g->lattice, cinv);
    std::vector<double> up(8 * n + 18);
    double *u_pos = up.data(), *u_q = u_pos + 3 * n, *u_frac = u_q + n, *u_scale = u_frac + 3 * n, *u_lat = u_scale + n,
           *u_cinv = u_lat + 9;
    std::copy(wpos.begin(), wpos.end(), u_pos);
    std::copy(q.begin(), q.end(), u_q);
    std::copy(frac.begin(), frac.end(), u_frac);
    for (int a = 0; a < nat; ++a) u_scale[a] = -q[a] * 4.0 * M_PI / g->dV;
    std::copy(g->lattice, g->lattice + 9, u_lat);
    std::copy(cinv, cinv + 9, u_cinv);
    std::vector<int> ui(start);
    ui.insert(ui.end(), order_atoms.begin(), order_atoms.end());
    ui.insert(ui.end(), cellof.begin(), cellof.end());
    double* d_up = (double*)sc.get("ew_up", up.size() * sizeof(double));
    int* d_ui = (int*)sc.get("ew_ui", ui.size() * sizeof(int));
    OFDFT_CK(cudaMemcpyAsync(d_up, up.data(), up.size() * sizeof(double), cudaMemcpyHostToDevice, st));
    OFDFT_CK(cudaMemcpyAsync(d_ui, ui.data(), ui.size() * sizeof(int), cudaMemcpyHostToDevice, st));
    double *d_pos = d_up, *d_q = d_pos + 3 * n, *d_frac = d_q + n, *d_scale = d_frac + 3 * n, *d_lat = d_scale + n,
           *d_cinv = d_lat + 9;
    double* d_F = (double*)sc.get("ew_F", 6 * n * sizeof(double));  // real-space, then reciprocal forces
    cl.start = d_ui;
    cl.atoms = d_ui + ncell + 1;
    cl.cellof = cl.atoms + nat;
    const int ablk = (nat + RED_THREADS - 1) / RED_THREADS;
    double* d_part = (double*)sc.get("ew_part", (size_t)std::max(ablk * 7, g->red_blocks) * sizeof(double));
    double* d_sums = (double*)sc.get("ew_sums", 7 * n * sizeof(double));
    k_ewald_real<<<(nat + kRealWarps - 1) / kRealWarps, 32 * kRealWarps, 0, st>>>(d_pos, d_q, nat, d_lat, cl, Rcut, eta,
                                                                                 d_F, d_sums);
    OFDFT_LAUNCH_CHECK();
    k_ewald_real_sum<<<ablk, RED_THREADS, 0, st>>>(d_sums, nat, d_part);
    OFDFT_LAUNCH_CHECK();
    reduce_finalize<<<7, RED_THREADS, 0, st>>>(d_part, ablk, 7, 0ull, g->d_results);
    OFDFT_LAUNCH_CHECK();

    // ---- reciprocal space
    // results: [0, 7) real-space sums, 7 the reciprocal energy, [8, 14) the reciprocal stress
    double e_rec = 0.0;
    double s_rec[6] = {0, 0, 0, 0, 0, 0};
    std::vector<double> Fall(6 * n, 0.0);
    const size_t cb = g->cplx_bytes(), rb = g->real_bytes();
    if (pme) {
        OFDFT_REQUIRE(g->nr[0] >= order && g->nr[1] >= order && g->nr[2] >= order,
                      "PME needs at least %d grid points per axis", order);
        std::vector<double> bm, bi;
        bspline_tables(g, order, bm, bi);
        const size_t nb = bm.size();
        bm.insert(bm.end(), bi.begin(), bi.end());
        double* bre = (double*)sc.get("ew_b", bm.size() * sizeof(double));
        double* bim = bre + nb;
        OFDFT_CK(cudaMemcpyAsync(bre, bm.data(), bm.size() * sizeof(double), cudaMemcpyHostToDevice, st));
        // two meshes: the charges, then the energy's terms, then the convolution; and their
        // transform, which becomes the convolution's in place
        const size_t mesh = std::max(rb, (size_t)g->Nc * sizeof(double2));
        Scratch& big = mesh + cb > kKeep ? own : sc;
        T* Q = (T*)big.get("ew_Q", mesh);
        C* QG = (C*)big.get("ew_QG", cb);
        double2* terms = reinterpret_cast<double2*>(Q);
        pme_spread<T>(sc, "ew_", nat, order, d_frac, nullptr, d_q, g->geo, Q, st);
        g->exec_r2c(Q, QG, 1, st);
        if (stress) {
            k_ewald_stress_rec<T><<<g->red_blocks, RED_THREADS, 0, st>>>(QG, nullptr, bre, bim, g->geo, eta,
                                                                         g->d_partials);
            OFDFT_LAUNCH_CHECK();
            reduce_finalize<<<6, RED_THREADS, 0, st>>>(g->d_partials, g->red_blocks, 6, 0ull, g->d_results + 8);
            OFDFT_LAUNCH_CHECK();
        }
        k_ewald_rec_pme<T><<<row_grid(g->geo, g->sms), 32 * kRowWarps, 0, st>>>(QG, forces != nullptr, bre, bim, g->geo,
                                                                                eta, terms);
        OFDFT_LAUNCH_CHECK();
        k_ewald_rec_sum<<<g->red_blocks, RED_THREADS, 0, st>>>(terms, g->Nc, d_part);
        OFDFT_LAUNCH_CHECK();
        reduce_finalize<<<1, RED_THREADS, 0, st>>>(d_part, g->red_blocks, 1, 0ull, g->d_results + 7);
        OFDFT_LAUNCH_CHECK();
        if (forces) {
            T* conv = Q;  // charges and terms are done with
            if (sizeof(T) == 8 && fix::grid_plans(g)) {
                double2* in = (double2*)QG;
                double* out = (double*)conv;
                fix::c2r(g, &in, &out, 1, st);
            } else {
                g->exec_c2r(QG, conv, 1, st);
            }
            k_pme_gather<T><<<nat, kGatherThreads, 0, st>>>(d_frac, nullptr, order, g->geo, conv, d_cinv, d_scale,
                                                            d_F + 3 * n);
            OFDFT_LAUNCH_CHECK();
        }
        OFDFT_CK(cudaMemcpyAsync(g->h_results, g->d_results, 14 * sizeof(double), cudaMemcpyDeviceToHost, st));
        if (forces)
            OFDFT_CK(cudaMemcpyAsync(Fall.data(), d_F, 6 * n * sizeof(double), cudaMemcpyDeviceToHost, st));
        OFDFT_CK(cudaStreamSynchronize(st));
        e_rec = 4.0 * M_PI * g->h_results[7] / g->volume;
        for (int k = 0; k < 6; ++k) s_rec[k] = stress ? g->h_results[8 + k] : 0.0;
    } else {
        OFDFT_CK(cudaMemcpyAsync(Fall.data(), d_F, 3 * n * sizeof(double), cudaMemcpyDeviceToHost, st));
        const size_t sb = (size_t)g->Nc * 2 * sizeof(double);
        double* S = (double*)(sb > kKeep / 2 ? own : sc).get("ew_S", sb);
        k_ewald_rec_exact<T><<<g->red_blocks, RED_THREADS, 0, st>>>(d_pos, d_q, nat, g->geo, eta, S, g->d_partials);
        OFDFT_LAUNCH_CHECK();
        reduce_finalize<<<1, RED_THREADS, 0, st>>>(g->d_partials, g->red_blocks, 1, 0ull, g->d_results + 7);
        OFDFT_LAUNCH_CHECK();
        OFDFT_CK(cudaMemcpyAsync(g->h_results, g->d_results, 8 * sizeof(double), cudaMemcpyDeviceToHost, st));
        OFDFT_CK(cudaStreamSynchronize(st));
        e_rec = 4.0 * M_PI * g->h_results[7] / g->volume;
        if (stress) {
            k_ewald_stress_rec<T><<<g->red_blocks, RED_THREADS, 0, st>>>(nullptr, S, nullptr, nullptr, g->geo, eta,
                                                                         g->d_partials);
            OFDFT_LAUNCH_CHECK();
            reduce_finalize<<<6, RED_THREADS, 0, st>>>(g->d_partials, g->red_blocks, 6, 0ull, g->d_results + 8);
            OFDFT_LAUNCH_CHECK();
            OFDFT_CK(cudaMemcpyAsync(s_rec, g->d_results + 8, 6 * sizeof(double), cudaMemcpyDeviceToHost, st));
            OFDFT_CK(cudaStreamSynchronize(st));
        }
        if (forces) {
            for (int a0 = 0; a0 < nat; a0 += kChunk) {
                const int na = std::min(kChunk, nat - a0);
                k_ewald_force_exact<<<g->red_blocks, RED_THREADS, 0, st>>>(d_pos, d_q, S, a0, na, g->geo, eta,
                                                                           g->d_partials);
                OFDFT_LAUNCH_CHECK();
                reduce_finalize<<<3 * kChunk, RED_THREADS, 0, st>>>(g->d_partials, g->red_blocks, 3 * kChunk, 0ull,
                                                           g->d_results + 16);
                OFDFT_LAUNCH_CHECK();
                OFDFT_CK(cudaMemcpyAsync(g->h_results + 16, g->d_results + 16, 3 * kChunk * sizeof(double),
                                         cudaMemcpyDeviceToHost, st));
                OFDFT_CK(cudaStreamSynchronize(st));
                for (int t = 0; t < na; ++t)
                    for (int c = 0; c < 3; ++c)
                        Fall[3 * (n + a0 + t) + c] = g->h_results[16 + 3 * t + c] * 8.0 * M_PI / g->volume;
            }
        }
    }
    const double e_real = g->h_results[0] / 2.0;
    double s_real[6];
    for (int k = 0; k < 6; ++k) s_real[k] = g->h_results[1 + k] * (-0.5 / g->volume);
    out_energy[0] = e_corr + e_real + e_rec;
    out_energy[1] = e_real;
    out_energy[2] = e_rec;
    out_energy[3] = e_corr;
    if (forces)
        for (size_t k = 0; k < 3 * n; ++k) forces[k] = Fall[k] + Fall[3 * n + k];
    if (stress) {
        // both reciprocal forms reduce to 4 pi / V^2 times the mask sums (the PME
        // form's 2 x 2 pi / V^2 / dV^2 with the dV^2 of its transforms); the G = 0
        // term (sum q)^2 4 pi / (8 eta V^2) sits on the diagonal
        const double V2 = g->volume * g->volume;
        const double sg0 = qs * qs * 4.0 * M_PI * (1.0 / (4.0 * eta * V2) / 2.0);
        static const int I[6] = {0, 0, 0, 1, 1, 2}, J[6] = {0, 1, 2, 1, 2, 2};
        for (int k = 0; k < 6; ++k) {
            double v = s_real[k] + s_rec[k] * 4.0 * M_PI / V2;
            if (I[k] == J[k]) v += sg0;
            stress[3 * I[k] + J[k]] = stress[3 * J[k] + I[k]] = v;
        }
    }
}

}  // namespace

// both precisions run the Ewald sums in float64: an FP32 grid gets a float64
// twin for the PME mesh, built for this call only
static void ewald_any(ofdft_grid* g, int nat, const double* pos, const double* charges, double precision, int pme,
               int bspline_order, double* out_energy, double* forces, double* out_eta, double* stress,
               cudaStream_t st) {
    OFDFT_REQUIRE(g && pos && charges && nat >= 1, "ofdft_ewald: bad argument");
    OFDFT_REQUIRE(precision > 0.0 && precision < 1.0, "ofdft_ewald: precision must be in (0, 1)");
    OFDFT_REQUIRE(!pme || (bspline_order >= 3 && bspline_order <= kMaxOrder), "B-spline order must be 3..%d",
                  kMaxOrder);
    if (g->prec == OFDFT_F64) {
        ewald_t<double>(g, nat, pos, charges, precision, pme, bspline_order, out_energy, forces, out_eta, stress, st);
        return;
    }
    ofdft_grid* gd = nullptr;
    int rc = ofdft_grid_create(g->nr, g->lattice, OFDFT_F64, &gd);
    if (rc != OFDFT_OK) throw Error{rc};
    try {
        ewald_t<double>(gd, nat, pos, charges, precision, pme, bspline_order, out_energy, forces, out_eta, stress, st);
    } catch (...) {
        ofdft_grid_destroy(gd);
        throw;
    }
    ofdft_grid_destroy(gd);
}

extern "C" int ofdft_ewald(ofdft_grid* g, int nat, const double* pos, const double* charges, double precision, int pme,
                           int bspline_order, double* out_energy, double* forces, double* out_eta, ofdft_stream s) {
    return guard([&] {
        OFDFT_REQUIRE(out_energy, "ofdft_ewald: null energy output");
        ewald_any(g, nat, pos, charges, precision, pme, bspline_order, out_energy, forces, out_eta, nullptr,
                  (cudaStream_t)s);
    });
}

extern "C" int ofdft_ewald_stress(ofdft_grid* g, int nat, const double* pos, const double* charges, double precision,
                                  int pme, int bspline_order, double* stress, double* out_eta, ofdft_stream s) {
    return guard([&] {
        OFDFT_REQUIRE(stress, "ofdft_ewald_stress: null stress output");
        double energy[4];
        ewald_any(g, nat, pos, charges, precision, pme, bspline_order, energy, nullptr, out_eta, stress,
                  (cudaStream_t)s);
    });
}
