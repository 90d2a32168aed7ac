// Float64 evaluation of TF, vW, LDA, Hartree, the local pseudopotential and the
// Wang-Teter term with integer-pipe transforms (fix_fft.cuh, fix_3d.cuh).
//
// The same quantities as the evaluator's general path (total.cu), arranged for a GPU
// whose float64 pipe is the bound of everything:
//   k_pre       every power of rho from one sixth root
//   rows, cols  the forward transforms of rho, sqrt(rho), rho^beta (rho^alpha) in
//               one launch per axis
//   k_cols_mul  axis 0 forward, 4 pi/G^2 | G^2/2 | K(G), axis 0 inverse in one launch
//   k_post      potential and energies, one reciprocal per point
#include "fix_eval.h"

#include "fix_3d.cuh"
#include "pointwise.cuh"

#include <algorithm>
#include <cmath>

using namespace ofdft;
using namespace ofdft::fix;

namespace {

// The range where float32 seeds hold, 2^-99 to 2^99 (also: not zero, negative or NaN).  From the
// high word: a float64 comparison takes a slot of the float64 pipe.
__device__ __forceinline__ bool ordinary(double x) {
    return (unsigned)(__double2hiint(x) - ((1023 - 99) << 20)) < (198u << 20);
}
__device__ __forceinline__ bool positive(double x) { return __double_as_longlong(x) > 0; }  // true for NaN, too

// 1/x of an ordinary x: a float32 seed y and one cubic Newton step
// y (1 + e + e^2), e = 1 - x y.  Two conversions and three float64 operations, where
// the division takes about ten.
__device__ __forceinline__ double recip(double x) {
    const double y = (double)__frcp_rn((float)x);
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

// The powers of a density that the pre-pass needs, every one within 0.51 units in the last place.
// v = x^(-1/6) = v0 (1 + d) with a float32 seed v0, whose square is exact in float64: the power
// x v0^k is taken as a sum of two float64 numbers, e = 1 - x v0^6 gives d by the binomial series
// of (1 - e)^(-1/6) (|e| below 1e-6), and (1 + d)^k - 1 corrects the power before its only
// rounding.  About 40 float64 operations for all of them; separate roots with products of them
// took as many and were off by 2 to 8 units, as the factors' roundings add up.
struct Roots {
    double c, c2, w, v, sq;  // x^(1/3), x^(2/3), x^(-1/3), x^(-1/6), x^(1/2)
    double r53;              // x^(5/3)
    double p56;              // x to the float64 number nearest 5/6
};
__device__ __forceinline__ Roots roots_of(double x) {
    Roots o;
    if (ordinary(x)) {
        const float xf = (float)x;
        const double v0 = (double)sqrtf(rcbrtf(xf)), a = v0 * v0;
        const double y = x * a, yl = fma(x, a, -y);               // x v0^2
        const double z = y * a, zl = fma(yl, a, fma(y, a, -z));   // x v0^4
        const double s = y * v0, sl = fma(yl, v0, fma(y, v0, -s));  // x v0^3
        const double p = x * v0, pl = fma(x, v0, -p);
        const double e = fma(-zl, a, fma(-z, a, 1.0));
        const double d = e * fma(e, 7.0 / 72.0, 1.0 / 6.0);
        const double d2 = fma(d, d, d + d), d3 = fma(d2, d, d2 + d), d4 = fma(d2, d2, d2 + d2);
        const double t = fma(y, d2, yl);
        o.v = fma(v0, d, v0);
        o.w = fma(a, d2, a);
        o.c2 = y + t;
        o.c = z + fma(z, d4, zl);
        o.sq = s + fma(s, d3, sl);
        const double h = x * y;
        o.r53 = h + fma(x, t, fma(x, y, -h));
        // the exponent is 3.7e-17 above 5/6
        const double more = (double)(3.700743415417188e-17f * __logf(xf));
        o.p56 = p + fma(p, d + more, pl);
    } else {
        o.c = cbrt(x);
        if (o.c < 1e-30) o.c = 1e-30;  // for LDA (xc/semilocal_xc.py:283-319), which alone takes c, w and v
        o.c2 = cbrt(x * x);
        o.w = 1.0 / o.c;
        o.v = sqrt(o.w);
        o.sq = sqrt(x > 0.0 ? x : 1e-30);  // kedf/vw.py:34-44
        o.r53 = x * o.c2;
        o.p56 = 0.0;  // not used
    }
    return o;
}

struct LdaRoots {
    double rs, srs, ex, vx;  // cbrt(3/(4 pi)), its square root, exchange prefactors
};

// Slater exchange + PZ81 correlation (xc/semilocal_xc.py:283-319) from the roots of r:
// sqrt(Rs) = sqrt(rs) r^(-1/6)
__device__ __forceinline__ void lda_roots(const Roots& p, const LdaRoots& k, double& ex, double& vx) {
    const double a = 0.0311, b = -0.048, c = 0.0020, d = -0.0116, g = -0.1423, b1 = 1.0529, b2 = 0.3334;
    const double Rs = k.rs * p.w;
    if (__double2hiint(Rs) < 0x3ff00000) {  // Rs < 1; NaN is not
        const double lr = log(Rs);
        ex = k.ex * p.c + (a * lr + b + c * Rs * lr + d * Rs);
        vx = k.vx * p.c + (lr * (a + (2.0 / 3) * c * Rs) + b - (1.0 / 3) * a + (1.0 / 3) * (2 * d - c) * Rs);
    } else {
        const double sRs = k.srs * p.v;
        const double inv = recip(1.0 + b1 * sRs + b2 * Rs);
        ex = k.ex * p.c + g * inv;
        vx = k.vx * p.c + (g + (7.0 / 6.0 * g * b1) * sRs + (4.0 / 3.0 * g * b2) * Rs) * (inv * inv);
    }
}

// NS block sums at partials[blockIdx.x * NS + s], a fixed tree per slot
template <int NS>
__device__ __forceinline__ void block_sums(double (&v)[NS], double* partials) {
    block_sum_store<NS>(v, partials);
}

struct PreK {
    const double* rho;
    const double* vloc;
    double* V;
    double* sq;
    double* rb;
    double* ra;
    double* kf;
    long long N;
    int tf, xc;
    int b56;  // beta = 5/6
    double tf_x, alpha, beta, cE, cV, threepi2;
    LdaRoots lda;
};

// Pointwise pre-pass: bound by the float64 pipe, 87% busy (128^3 with TF, LDA, PP, vW and
// rho^(5/6), which needs no pow(): 264 us).
// LWT: also k_F and its range (three more slots, after all blocks' sums), and LWT's clamp.
template <bool LWT>
__global__ void __launch_bounds__(RED_THREADS) k_pre(PreK a, double* partials) {
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    double mm[3] = {INFINITY, -INFINITY, -INFINITY};
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < a.N; i += stride) {
        const double r = a.rho[i];
        double v = 0.0;
        s[3] += r;
        const Roots p = roots_of(r);
        if (a.tf) {
            s[0] += p.r53 * a.cE;
            v = a.cV * p.c2 * a.tf_x;
        }
        if (a.xc) {
            double ex, vx;
            lda_roots(p, a.lda, ex, vx);
            s[1] += ex * r;
            v += vx;
        }
        if (a.vloc) {
            const double vl = a.vloc[i];
            s[2] += vl * r;
            v += vl;
        }
        if (a.sq) a.sq[i] = p.sq;
        if (a.rb) {
            // wt.py:15-18; lwt.py:206-221
            const double rc = LWT ? (r > 0.0 ? r : 1e-30) : (r < kZERO ? kZERO : r);
            a.rb[i] = a.b56 && ordinary(r) ? p.p56 : pow(rc, a.beta);
            if (a.ra) a.ra[i] = pow(rc, a.alpha);
        }
        if (LWT) {
            // lwt.py:106.  To the last bit as the general path has it: a point at a node's k_F is
            // inside an interval or, at the last node, outside every one
            const double kf = 2.0 * cbrt(a.threepi2 * r);
            a.kf[i] = kf;
            mm[0] = fmin(mm[0], kf);
            mm[1] = fmax(mm[1], kf);
            mm[2] = fmax(mm[2], r);
        }
        if (a.V) a.V[i] = v;
    }
    block_sums<4>(s, partials);
    if (LWT) {
        const int kinds[3] = {1, 2, 2};
        block_reduce_store<3>(mm, kinds, partials + 4 * (long long)gridDim.x);
    }
}

// Block sums of ns slots into out[0..ns), in a fixed order, and (plan != 0) the
// Wang-Teter kernel state (wt.py:58-73: rebuilt when rho0 moves by more than 1e-6)
__global__ void k_sums(const double* __restrict__ partials, int nblk, int ns, double* out, int plan, double* state,
                       double rho0_fixed, double invN, double alpha, double beta, double cTF) {
    const int lane = threadIdx.x & 31, s = threadIdx.x >> 5;
    __shared__ double sh[4];
    if (s < ns) {
        double x = 0.0;
#pragma unroll 4
        for (int b = lane; b < nblk; b += 32) x += partials[(long long)b * ns + s];
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if (lane == 0) out[s] = sh[s] = x;
    }
    __syncthreads();
    if (plan && threadIdx.x == 0) {
        const double rho0 = rho0_fixed > 0.0 ? rho0_fixed : sh[3] * invN;
        if (state[4] == 0.0 || fabs(state[0] - rho0) > 1e-6) {
            state[0] = rho0;
            state[1] = 1.0;
            state[2] = 2.0 * pow(3.0 * rho0 * (M_PI * M_PI), 1.0 / 3.0);
            state[3] = 5.0 / (9.0 * alpha * beta * pow(rho0, alpha + beta - 5.0 / 3.0)) * cTF;
            state[4] = 1.0;
        } else {
            state[1] = 0.0;
        }
    }
}

enum { F_HARTREE = 0, F_VW = 1, F_WT = 2 };

struct MulArgs {
    ColArgs c;
    int kind[kMaxFields];
    Geo geo;
    double* K;  // Wang-Teter kernel
    const double* state;
    double wt_x, invN;
};

__device__ __noinline__ double wt_build(const MulArgs& a, double gg) {
    return lindhard_dev(sqrt(gg) / a.state[2], a.wt_x, 1.0) * a.state[3];
}

// The last pass of a forward transform, the factor, and the first pass of the inverse with
// the radices in reverse order: that one takes exactly the elements that this one leaves in
// a thread's registers, so they are not exchanged in between.
template <int R, class Factor>
__device__ __forceinline__ void turn(const I2* src, I2* dst, const Plan& p, int lb, LineSm& sm, Factor factor) {
    const int L = 1 << lb, m = p.n / R, l = threadIdx.x & (L - 1), j = threadIdx.x >> lb;
    const bool on = j < m;
    I2 u[R];
    double2 v[R];
    if (on) {
        gather<R>(u, src, p.n, lb, m, j, l, pass_shift(sm.ds[l], p.np - 1, p.np, p.r[1]), p.tw);
        Dft<R>::run(u);
#pragma unroll
        for (int q = 0; q < R; ++q) {
            const double2 z = from_fix(u[q], sm, l);
            const double f = factor(j + q * m);
            v[q] = make_double2(z.y * f, z.x * f);  // parts exchanged: the inverse
        }
    }
    __syncthreads();  // the buffer and the scales are read
    reset(sm);
    __syncthreads();
    agree<R>(v, u, on, j, l, sm, p.np);
    if (on) {
        Dft<R>::run(u);
#pragma unroll
        for (int q = 0; q < R; ++q) dst[(j * R + q) * (L + 1) + l] = u[q];
    }
}

// Axis 0 forward, the field's factor, axis 0 inverse.  G = f0 b0 + c along a line (f0 the axis-0
// frequency), |G|^2 the sum of its squares: six operations.  As a polynomial in f0, in two, it
// lost up to 150 units in cells whose reciprocal vectors nearly cancel.
__global__ void __launch_bounds__(kThreads, kBlocks) k_cols_mul(MulArgs a) {
    extern __shared__ __align__(16) unsigned char fix_smem[];
    __shared__ LineSm sm;
    const Plan& p = a.c.g.p0;
    const int n = p.n, lb = a.c.lb, L = 1 << lb;
    I2* b0 = reinterpret_cast<I2*>(fix_smem);
    I2* b1 = b0 + (p.np == 3 ? n * (L + 1) : 0);
    double* fq = reinterpret_cast<double*>(b1 + n * (L + 1));  // f0
    const int line = (blockIdx.x << lb) + (threadIdx.x & (L - 1));
    const bool in = line < col_lines<0>(a.c.g);
    const int k1 = line / a.c.g.n2h, k2 = line - k1 * a.c.g.n2h;
    const long long stride = col_stride<0>(a.c.g);
    double2* base = a.c.sp[blockIdx.y] + (in ? line : 0);
    const int kind = a.kind[blockIdx.y];
    const Geo& g = a.geo;
    const double f1 = (double)freq_index(k1, g.n1) * g.fv[1], f2 = (double)k2 * g.fv[2];
    const double cx = f1 * g.b[3] + f2 * g.b[6], cy = f1 * g.b[4] + f2 * g.b[7], cz = f1 * g.b[5] + f2 * g.b[8];
    auto gsq_at = [&](int i) {
        const double f = fq[i], gx = fma(f, g.b[0], cx), gy = fma(f, g.b[1], cy), gz = fma(f, g.b[2], cz);
        return fma(gx, gx, fma(gy, gy, gz * gz));
    };
    for (int i = threadIdx.x; i < n; i += blockDim.x) fq[i] = (double)freq_index(i, n) * g.fv[0];
    const bool build = kind == F_WT && a.state[1] != 0.0;
    const double hart = 4.0 * M_PI * a.invN, half = 0.5 * a.invN;
    auto factor = [&](int i) -> double {
        if (!in) return 0.0;
        if (kind == F_WT) {
            const long long at = line + i * stride;
            if (!build) return a.K[at] * a.invN;
            const double K = wt_build(a, gsq_at(i));
            a.K[at] = K;
            return K * a.invN;
        }
        const double gg = gsq_at(i);
        if (kind == F_VW) return gg * half;
        return i == 0 && line == 0 ? 0.0 : (ordinary(gg) ? recip(gg) : 1.0 / gg) * hart;
    };
    auto get = [&](int i, int) { return in ? base[i * stride] : make_double2(0.0, 0.0); };
    auto put = [&](int i, int l, I2 z) {
        if (in) base[i * stride] = swapped(from_fix(z, sm, l));
    };
    reset(sm);
    __syncthreads();
    switch (p.r[0]) {
#define FIX_CASE(R) \
    case R: pass0<R>(b0, n, lb, sm, p.np, get); break;
        FIX_RADICES(FIX_CASE)
#undef FIX_CASE
    }
    __syncthreads();
    if (p.np == 1) {  // one pass: the transform's outputs are in the buffer
        const int l = threadIdx.x & (L - 1), k = sm.ds[l] - sm.k[l];
        const bool nan = sm.emax[l] == kNonFinite;
        __syncthreads();
        tile_fft_out(
            b0, b1, p, lb, sm,
            [&](int i, int q) {
                const I2 z = b0[i * (L + 1) + q];
                const double f = factor(i);
                return make_double2(to_dbl(z.y, k, nan) * f, to_dbl(z.x, k, nan) * f);
            },
            put);
        return;
    }
    const I2* z = middle(b0, b1, p, lb, sm, p.np - 1, false);
    I2* y = z == b0 ? b0 : b1;
    switch (p.r[p.np - 1]) {
#define FIX_CASE(R) \
    case R: turn<R>(z, y, p, lb, sm, factor); break;
        FIX_RADICES(FIX_CASE)
#undef FIX_CASE
    }
    __syncthreads();
    z = middle(y, y == b0 ? b1 : b0, p, lb, sm, p.np - 1, true);
    switch (p.r[0]) {
#define FIX_CASE(R) \
    case R: pass_out<R>(z, n, lb, p.tw, sm, p.np - 1, p.np, p.r[p.np - 2], put); break;
        FIX_RADICES(FIX_CASE)
#undef FIX_CASE
    }
}

struct PostK {
    const double* rho;
    double* V;
    const double* sq;
    const double* lap;
    const double* vH;
    const double* nl1;
    const double* nl2;
    const double* rb;
    const double* ra;
    long long N;
    double vw_y, alpha, beta, half_alpha;  // 0.5 / alpha
    // density-dependent kernel
    const double* kf;
    const double* pot1[4];
    const double* pot2;
    const double* pot3[4];
    double rhomax, ld, kfclip;
};

// Pointwise post-pass: vW and Hartree potentials, the Wang-Teter potential
// (wt.py:19-23, 44-56, 124-132) and their energies.  Float64 pipe 83% busy (128^3: 99 us)
__global__ void __launch_bounds__(RED_THREADS) k_post(PostK a, double* partials) {
    double s[3] = {0.0, 0.0, 0.0};
    const double tiny = 1e-30;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < a.N; i += stride) {
        const double r = a.rho[i];
        const bool ord = ordinary(r);
        const double ri = ord ? recip(r) : 1.0 / (r < kZERO ? kZERO : r);
        double v = a.V ? a.V[i] : 0.0;
        if (a.lap) {
            double q = a.sq[i];
            if (!ord && fabs(q) < tiny) q = tiny;
            const double pw = a.lap[i] * (ord ? q * ri : 1.0 / q);
            if (positive(r)) s[0] += r * pw;
            v += pw * a.vw_y;
        }
        if (a.vH) {
            const double vh = a.vH[i];
            s[1] += vh * r;
            v += vh;
        }
        if (a.nl1) {
            const double pb = a.rb[i], c1 = a.nl1[i];
            if (!a.ra) {
                const double pot = 2.0 * a.alpha * (pb * ri) * c1;
                if (a.V) s[2] += pot * r * a.half_alpha;
                else s[2] += c1 * pb;
                v += pot;
            } else {
                const double pa = a.ra[i];
                s[2] += c1 * pa;
                if (a.V) v += a.alpha * (pa * ri) * c1 + a.beta * (pb * ri) * a.nl2[i];
            }
        }
        if (a.pot1[0]) {
            auto parts = [&](const double* const (&p)[4]) {  // null: no part
                double x = 0.0;
                for (int k = 0; k < 4; ++k)
                    if (p[k]) x += p[k][i];
                return x;
            };
            // low-density factor (lwt.py:315-322) and the combination (:324-339)
            double f = 1.0;
            if (r < 1e-6) f = pow(fabs(r), a.ld) / pow(a.rhomax, a.ld);
            if (r < 0.0) f = 0.0;
            const double rc = ord ? ri : 1.0 / (r > 0.0 ? r : tiny);
            const double pa = a.ra ? a.ra[i] : a.rb[i], p1 = parts(a.pot1) * f;
            s[2] += pa * p1;
            if (a.V) {
                const double p2 = a.pot2 ? a.pot2[i] * f : p1;
                const double p3 = parts(a.pot3) * f;
                const double kf = fmin(a.kf[i], a.kfclip);
                v += a.alpha * (pa * rc) * p1 + (a.beta * (a.rb[i] * rc) * p2 + kf * (1.0 / 3.0) * (pa * rc) * p3);
            }
        }
        if (a.V) a.V[i] = v;
    }
    block_sums<3>(s, partials);
}

}  // namespace

namespace ofdft {
namespace fix {

struct GridPlans {
    Grid3 g;
    Tw* tw = nullptr;
    bool ok = false;
};

const Grid3* grid_plans(ofdft_grid* g) {
    if (g->prec != OFDFT_F64) return nullptr;
    if (!g->fix) {
        GridPlans* h = new GridPlans();
        g->fix = h;
        h->g.n0 = g->nr[0];
        h->g.n1 = g->nr[1];
        h->g.n2 = g->nr[2];
        h->g.n2h = g->n2h;
        Plan* p[3] = {&h->g.p0, &h->g.p1, &h->g.p2};
        bool ok = true;
        size_t total = 0;
        for (int d = 0; d < 3; ++d) {
            ok = ok && plan_radices(g->nr[d], *p[d]);
            total += (size_t)g->nr[d];
        }
        if (ok) {
            // twiddles at scale 2^61 from long double trigonometry
            std::vector<Tw> tw(total);
            size_t off = 0;
            const long double pi = 3.14159265358979323846264338327950288L;
            for (int d = 0; d < 3; ++d) {
                const int n = g->nr[d];
                for (int k = 0; k < n; ++k) {
                    const long double t = -2.0L * pi * (long double)k / (long double)n;
                    tw[off + k] = tw_of((long long)std::llroundl(std::cos(t) * (long double)kOne),
                                        (long long)std::llroundl(std::sin(t) * (long double)kOne));
                }
                off += n;
            }
            OFDFT_CK(cudaMalloc(&h->tw, total * sizeof(Tw)));
            upload_now(h->tw, tw.data(), total * sizeof(Tw));
            off = 0;
            for (int d = 0; d < 3; ++d) {
                p[d]->tw = h->tw + off;
                off += g->nr[d];
            }
            h->ok = true;
        }
    }
    const GridPlans* h = static_cast<const GridPlans*>(g->fix);
    return h->ok ? &h->g : nullptr;
}

void free_plans(ofdft_grid* g) {
    GridPlans* h = static_cast<GridPlans*>(g->fix);
    if (!h) return;
    if (h->tw) cudaFree(h->tw);
    delete h;
    g->fix = nullptr;
}

void r2c(ofdft_grid* g, const double* const* in, double2* const* out, int nf, cudaStream_t st) {
    const Grid3& p = *grid_plans(g);
    rows_r2c(p, g->sms, in, out, nf, st);
    cols<1>(p, g->sms, out, nf, false, st);
    cols<0>(p, g->sms, out, nf, false, st);
}

void c2r(ofdft_grid* g, double2* const* in, double* const* out, int nf, cudaStream_t st) {
    const Grid3& p = *grid_plans(g);
    cols<0>(p, g->sms, in, nf, true, st);
    cols<1>(p, g->sms, in, nf, true, st);
    rows_c2r(p, g->sms, in, out, nf, st);
}

static int point_blocks(const ofdft_grid* g) {
    return (int)std::max(1LL, std::min((long long)g->sms * 8, (g->N + RED_THREADS - 1) / RED_THREADS));
}

int local_begin(ofdft_grid* g, Scratch& sc, const LocalArgs& a, Fields& f, cudaEvent_t copied, cudaStream_t st) {
    const Grid3& p = *grid_plans(g);
    const long long N = g->N;
    const size_t rb = g->real_bytes(), cb = g->cplx_bytes();
    const int sms = g->sms;
    const bool nl = a.wt || a.lwt, same = std::fabs(a.beta - a.alpha) < (a.wt ? 1e-9 : 1e-8);
    f.sq = a.vw ? (double*)sc.get("sq", rb) : nullptr;
    f.rb = nl ? (double*)sc.get("rb", rb) : nullptr;
    f.ra = nl && !same ? (double*)sc.get("ra", rb) : nullptr;
    f.kf = a.lwt ? (double*)sc.get("kf", rb) : nullptr;
    const int blocks = point_blocks(g);
    double* part = (double*)sc.get("fix_part", (size_t)blocks * 7 * sizeof(double));
    const Consts k = make_consts();

    PreK pk{};
    pk.rho = a.rho;
    pk.vloc = a.vloc;
    pk.V = a.V;
    pk.sq = f.sq;
    pk.rb = f.rb;
    pk.ra = f.ra;
    pk.kf = f.kf;
    pk.N = N;
    pk.tf = a.tf;
    pk.xc = a.xc;
    pk.b56 = a.beta == 5.0 / 6.0;
    pk.tf_x = a.tf_x;
    pk.alpha = a.alpha;
    pk.beta = a.beta;
    pk.cE = k.cTF_E;
    pk.cV = k.cTF_V;
    pk.threepi2 = k.threepi2;
    pk.lda = LdaRoots{k.lda_rs, std::sqrt(k.lda_rs), k.lda_ex, k.lda_vx};
    const double real = (double)rb, cplx = (double)cb;
    a.time(PRE, real * (1 + (a.vloc != nullptr) + (a.V != nullptr) + a.vw + nl + (f.ra != nullptr) + a.lwt), st, [&] {
        if (a.lwt) k_pre<true><<<blocks, RED_THREADS, 0, st>>>(pk, part);
        else k_pre<false><<<blocks, RED_THREADS, 0, st>>>(pk, part);
    });
    a.time(SUMS, blocks * 4.0 * sizeof(double), st, [&] {
        k_sums<<<1, 128, 0, st>>>(part, blocks, 4, g->d_results, a.wt, a.wtstate, a.wt_rho0, 1.0 / (double)N, a.alpha,
                                  a.beta, a.cTF_wt);
    });
    int launches = 2;
    if (a.lwt) {
        a.time(SUMS, blocks * 3.0 * sizeof(double), st, [&] {
            reduce_finalize<<<3, RED_THREADS, 0, st>>>(part + 4 * (size_t)blocks, blocks, 3,
                                                       1ull | (2ull << 2) | (2ull << 4), g->d_results + 4);
        });
        OFDFT_CK(cudaMemcpyAsync(g->h_results, g->d_results, 7 * sizeof(double), cudaMemcpyDeviceToHost, st));
        OFDFT_CK(cudaEventRecord(copied, st));
        ++launches;
    }

    // fields to transform, their factors and what they become
    const double* in[4];
    double2* sp[4];
    double* out[4];
    MulArgs m{};
    int nf = 0;
    auto field = [&](const double* src, const char* spec, const char* real, int kind) {
        in[nf] = src;
        sp[nf] = (double2*)sc.get(spec, cb);
        out[nf] = (double*)sc.get(real, rb);
        m.kind[nf] = kind;
        return out[nf++];
    };
    if (a.h) f.vH = field(a.rho, "rhoG", "vH", F_HARTREE);
    if (a.vw) f.lap = field(f.sq, "sqG", "lap", F_VW);
    if (a.wt) f.nl1 = field(f.rb, "rbG", "nl1", F_WT);
    if (a.wt && f.ra) f.nl2 = field(f.ra, "raG", "nl2", F_WT);
    const int back = nf;  // fields that are transformed back
    if (a.lwt) {
        in[nf] = f.rb;
        f.rbG = sp[nf++] = (double2*)sc.get("rbG", cb);
    }
    if (nf > 0) {
        a.time(FFT, nf * (real + cplx), st, [&] { rows_r2c(p, sms, in, sp, nf, st); });
        a.time(FFT, nf * 2 * cplx, st, [&] { cols<1>(p, sms, sp, nf, false, st); });
        launches += 2;
    }
    if (a.lwt) {
        a.time(FFT, 2 * cplx, st, [&] { cols<0>(p, sms, &f.rbG, 1, false, st); });
        ++launches;
    }
    if (back > 0) {
        const Shape s = shape_of(p.p0, col_lines<0>(p), sms, true);
        m.c.g = p;
        m.c.lb = s.lb;
        for (int i = 0; i < back; ++i) m.c.sp[i] = sp[i];
        m.geo = g->geo;
        m.K = a.wtK;
        m.state = a.wtstate;
        m.wt_x = a.wt_x;
        m.invN = 1.0 / (double)N;
        const size_t smem = tile_smem(p.p0, s.lb, 1) + (size_t)p.n0 * sizeof(double);
        smem_optin(k_cols_mul, smem);
        a.time(FFT, (back * 2 + (a.wt ? 0.5 : 0.0)) * cplx, st, [&] {
            k_cols_mul<<<dim3(col_blocks(col_lines<0>(p), s.lb), back), s.threads, smem, st>>>(m);
        });
        a.time(FFT, back * 2 * cplx, st, [&] { cols<1>(p, sms, sp, back, true, st); });
        a.time(FFT, back * (real + cplx), st, [&] { rows_c2r(p, sms, sp, out, back, st); });
        launches += 3;
    }
    return launches;
}

int local_finish(ofdft_grid* g, Scratch& sc, const LocalArgs& a, const Fields& f, const LwtPost& w, cudaStream_t st) {
    const int blocks = point_blocks(g);
    double* part = (double*)sc.get("fix_part", (size_t)blocks * 7 * sizeof(double));
    PostK q{};
    q.rho = a.rho;
    q.V = a.V;
    q.sq = f.sq;
    q.lap = f.lap;
    q.vH = f.vH;
    q.nl1 = f.nl1;
    q.nl2 = f.nl2;
    q.rb = f.rb;
    q.ra = f.ra;
    q.N = g->N;
    q.vw_y = a.vw_y;
    q.alpha = a.alpha;
    q.beta = a.beta;
    q.half_alpha = 0.5 / a.alpha;
    q.kf = f.kf;
    q.pot2 = w.pot2;
    for (int i = 0; i < 4; ++i) q.pot1[i] = w.pot1[i], q.pot3[i] = w.pot3[i];
    q.rhomax = w.rhomax;
    q.ld = w.ld;
    q.kfclip = w.kfclip;
    int fields = 1;  // read, and V written
    for (const void* x : {(const void*)f.sq, (const void*)f.lap, (const void*)f.vH, (const void*)f.nl1, (const void*)f.nl2,
                          (const void*)f.rb, (const void*)f.ra, (const void*)f.kf, (const void*)w.pot2})
        fields += x != nullptr;
    for (int i = 0; i < 4; ++i) fields += (w.pot1[i] != nullptr) + (w.pot3[i] != nullptr);
    fields += a.V ? 2 : 0;
    a.time(POST, (double)g->real_bytes() * fields, st, [&] { k_post<<<blocks, RED_THREADS, 0, st>>>(q, part); });
    a.time(SUMS, blocks * 3.0 * sizeof(double), st, [&] {
        k_sums<<<1, 128, 0, st>>>(part, blocks, 3, g->d_results + 16, 0, nullptr, 0.0, 0.0, 0.0, 0.0, 0.0);
    });
    return 2;
}

}  // namespace fix
}  // namespace ofdft
