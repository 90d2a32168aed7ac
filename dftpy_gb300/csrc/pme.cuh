// Smooth-PME building blocks shared by the local pseudopotential and Ewald:
// cardinal B-spline charge spreading, Q[l0(i), l1(j), l2(k)] += w_a M(i) M(j) M(k)
// with l_d(i) = (1 + floor(u_d) - i) mod n_d, u = frac * n (ewald.py:172-194),
// and the gradient gather for forces (src/dftpy/ewald.py:63-82, :137-194,
// :810-864; pseudo/__init__.py:523-571).
#pragma once
#include "common.cuh"

#include <algorithm>
#include <string>

namespace ofdft {

constexpr int kMaxOrder = 16;

__device__ inline int pmod(long long a, int n) {
    long long r = a % n;
    return (int)(r < 0 ? r + n : r);
}

// B-spline values M_order(x + n - 1), n = 1..order (ewald.py:63-82), with one lane per n: lane
// n - 1 of a group of 16 holds M_i(x + n - 1) after step i.  before: the values of order - 1
// (what the derivatives need).
__device__ __forceinline__ double bspline_mn_lane(double x, int order, int n, double& before) {
    double v = n == 1 ? x : (n == 2 ? 1.0 - x : 0.0);
    before = v;
    for (int i = 3; i <= order; ++i) {
        before = v;
        double below = __shfl_up_sync(0xffffffffu, v, 1, 16);
        if (n == 1) below = 0.0;
        const int j = i - n;
        double w = (x + n - 1) * v + (j + 1 - x) * below;
        w /= (double)(i - 1);
        v = n <= i ? w : 0.0;
    }
    return v;
}

// ---------------------------------------------------------------------------
// Deterministic spreading.  The grid is cut into 8 x 8 x 32 tiles, one block each, four grid
// points (8 apart on axis 2) per thread.  The block goes through the atoms in list order, 512
// at a time: every thread tests one atom's order^3 stencil against the tile, the hits are
// compacted in order into shared memory, and every thread sums their contributions in that
// order in float64 and stores its points once.  The sum at every point has a fixed order, so Q
// is the same bits on every run (a per-atom scatter with global atomics sums in arrival order).
// The test costs tiles x atoms comparisons and bounds the kernel, hence the long tiles (2048
// atoms on 256^3: 149 us; 8^3 tiles: 404 us); lists built and sorted on the host took 2.5 ms
// there.  From kPmeSlabAtoms atoms on, every slab of 8 points along axis 0 first gets the list of
// the atoms that touch it (the same order), and its tiles test those.  v_loc without and with the
// lists, ms: 108 atoms on 64^3 0.13 and 0.14; 4000 on 96^3 0.31 and 0.32, on 256^3 0.89 and 0.78;
// 16384 on 128^3 0.89 and 0.85, on 512^3 10.1 and 5.3; 131072 on 1024^3 378 and 43.
constexpr int kPmeTile = 8;
constexpr int kPmeLong = 4;  // 8-point pieces of a tile along axis 2
constexpr int kPmeThreads = kPmeTile * kPmeTile * kPmeTile;
constexpr int kPmeSlabAtoms = 4096;

// Stencil base and B-spline weights of every list position: 16 lanes per atom and axis
static __global__ void k_pme_prep(const double* __restrict__ frac, const int* __restrict__ list, int nlist, int order,
                                  Geo geo, int* base, double* M) {
    const int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 4, n = (threadIdx.x & 15) + 1;
    const bool on = g < 3 * nlist;
    const int q = on ? g / 3 : 0, d = on ? g - 3 * q : 0;
    const int a = list ? list[q] : q;
    const int nr = d == 0 ? geo.n0 : (d == 1 ? geo.n1 : geo.n2);
    const double up = frac[3 * a + d] * (double)nr;
    const double fl = floor(up);
    double before;
    const double v = bspline_mn_lane(up - fl, order, n, before);
    if (!on) return;
    double* out = M + (size_t)g * (order + 1);
    if (n <= order) out[n] = v;
    if (n == 1) {
        out[0] = 0.0;
        base[g] = (int)fl;
    }
}

// Whether the order points of an atom's stencil with base b along an axis of n points touch the
// `wide` points from lo on; t = (1 + b - lo) mod n
__device__ __forceinline__ bool pme_touches(int b, int lo, int n, int wide, int order, int& t) {
    t = 1 + b - lo;  // base in [0, n): t in (-n, n]
    t = t < 0 ? t + n : (t >= n ? t - n : t);
    return t <= order + min(wide, n - lo) - 2;
}

// Ordered lists of the atoms that touch each slab of 8 points along axis 0, one block per slab:
// counts, then (FILL) the lists one after another, with their starts.  An atom's points lie in
// at most pme_slabs_of(order) slabs: a run of them, cut where it wraps around or meets the axis's
// partial slab.
inline int pme_slabs_of(int order) { return order / kPmeTile + 4; }
template <bool FILL>
static __global__ void __launch_bounds__(kPmeThreads)
    k_pme_slabs(int nlist, int order, const int* __restrict__ base, int n0, int* __restrict__ counts,
                int* __restrict__ starts, int* __restrict__ lists, long long room) {
    __shared__ int part[kPmeThreads / 32];
    __shared__ int from;
    const int lo = blockIdx.x * kPmeTile, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) from = 0;
    __syncthreads();
    if (FILL) {
        int before = 0;
        for (int s = threadIdx.x; s < (int)blockIdx.x; s += kPmeThreads) before += counts[s];
        if (before) atomicAdd(&from, before);
        __syncthreads();
        if (threadIdx.x == 0) starts[blockIdx.x] = from;
    }
    int found = FILL ? from : 0;
    for (int q0 = 0; q0 < nlist; q0 += kPmeThreads) {
        const int q = q0 + threadIdx.x;
        int t;
        const bool on = q < nlist && pme_touches(base[3 * q], lo, n0, kPmeTile, order, t);
        const unsigned b = __ballot_sync(0xffffffffu, on);
        __syncthreads();  // part is read
        if (lane == 0) part[warp] = __popc(b);
        __syncthreads();
        int at = found;
        for (int k = 0; k < kPmeThreads / 32; ++k) {
            at += k < warp ? part[k] : 0;
            found += part[k];
        }
        if (FILL && on) {
            at += __popc(b & ((1u << lane) - 1u));
            if (at < room) lists[at] = q;
        }
    }
    if (!FILL && threadIdx.x == 0) counts[blockIdx.x] = found;
}

// Q at every point of a tile: sum over the atoms that touch it, in list order, of
// w_a M0(i) M1(j) M2(k) with i = (1 + base_0 - l0) mod n0 (< order), etc.  counts, starts,
// lists: of k_pme_slabs, or null
template <typename T>
__global__ void __launch_bounds__(kPmeThreads)
    k_pme_tiles(int nlist, int order, const int* __restrict__ base, const double* __restrict__ M,
                const double* __restrict__ w, const int* __restrict__ list, Geo geo, T* Q,
                const int* __restrict__ counts, const int* __restrict__ starts, const int* __restrict__ lists) {
    __shared__ int hit[kPmeThreads];
    __shared__ int off[kPmeThreads][3];  // (1 + base - first point of the tile) mod n per axis
    __shared__ int count[kPmeThreads / 32];
    const int T1 = (geo.n1 + kPmeTile - 1) / kPmeTile;
    constexpr int wide = kPmeTile * kPmeLong;
    const int T2 = (geo.n2 + wide - 1) / wide;
    const int tid = blockIdx.x, nr[3] = {geo.n0, geo.n1, geo.n2};
    const int lo[3] = {(tid / (T1 * T2)) * kPmeTile, ((tid / T2) % T1) * kPmeTile, (tid % T2) * wide};
    const int p[3] = {(int)(threadIdx.x >> 6), (int)((threadIdx.x >> 3) & 7), (int)(threadIdx.x & 7)};
    const bool in = lo[0] + p[0] < nr[0] && lo[1] + p[1] < nr[1] && lo[2] + p[2] < nr[2];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, o1 = order + 1;
    double v[kPmeLong] = {};
    const int slab = tid / (T1 * T2), atoms = lists ? counts[slab] : nlist;
    const int* mine = lists ? lists + starts[slab] : nullptr;
    for (int q0 = 0; q0 < atoms; q0 += kPmeThreads) {
        int q = q0 + threadIdx.x;
        int o[3] = {0, 0, 0};
        bool on = q < atoms;
        if (on) {
            if (mine) q = mine[q];
#pragma unroll
            for (int d = 0; d < 3; ++d)
                on = pme_touches(base[3 * q + d], lo[d], nr[d], d == 2 ? wide : kPmeTile, order, o[d]) && on;
        }
        const unsigned b = __ballot_sync(0xffffffffu, on);
        __syncthreads();  // the previous chunk's list is done with
        if (lane == 0) count[warp] = __popc(b);
        __syncthreads();
        int at = 0, total = 0;
#pragma unroll
        for (int k = 0; k < kPmeThreads / 32; ++k) {
            const int c = count[k];
            at += k < warp ? c : 0;
            total += c;
        }
        if (on) {
            at += __popc(b & ((1u << lane) - 1u));
            hit[at] = q;
            off[at][0] = o[0];
            off[at][1] = o[1];
            off[at][2] = o[2];
        }
        __syncthreads();
        if (!in) continue;
        for (int h = 0; h < total; ++h) {
            int i0 = off[h][0] - p[0], j0 = off[h][1] - p[1];
            i0 += i0 < 0 ? nr[0] : 0;
            j0 += j0 < 0 ? nr[1] : 0;
            if (i0 >= order || j0 >= order) continue;
            const int a = hit[h];
            const double* M0 = M + (3 * (size_t)a) * o1;
            const double* M1 = M0 + o1;
            const double* M2 = M1 + o1;
            const double wa = w ? w[list ? list[a] : a] : 1.0;
#pragma unroll
            for (int s = 0; s < kPmeLong; ++s) {
                int k0 = off[h][2] - p[2] - s * kPmeTile;
                k0 += k0 < 0 ? nr[2] : 0;
                // n >= order in practice; the loops also cover a stencil that wraps onto itself
                if (k0 >= 0 && k0 < order)
                    for (int i = i0; i < order; i += nr[0])
                        for (int j = j0; j < order; j += nr[1])
                            for (int k = k0; k < order; k += nr[2]) v[s] += wa * M0[i + 1] * M1[j + 1] * M2[k + 1];
            }
        }
    }
    if (!in) return;
    T* out = Q + ((long long)(lo[0] + p[0]) * geo.n1 + lo[1] + p[1]) * geo.n2;
#pragma unroll
    for (int s = 0; s < kPmeLong; ++s) {
        const int k = lo[2] + p[2] + s * kPmeTile;
        if (k < nr[2]) out[k] = (T)v[s];
    }
}

// Q = the spread of the list's atoms with weights w (null: 1).  d_frac, d_list and d_w on
// the device (d_list and d_w may be null); work buffers of sc named prefix + "...".
template <typename T>
void pme_spread(Scratch& sc, const std::string& prefix, int nlist, int order, const double* d_frac, const int* d_list,
                const double* d_w, const Geo& geo, T* Q, cudaStream_t st) {
    const size_t qbytes = (size_t)geo.N * sizeof(T);
    if (nlist <= 0) {
        OFDFT_CK(cudaMemsetAsync(Q, 0, qbytes, st));
        return;
    }
    int* base = (int*)sc.get(prefix + "base", 3 * (size_t)nlist * sizeof(int));
    double* M = (double*)sc.get(prefix + "M", 3 * (size_t)(order + 1) * nlist * sizeof(double));
    const int groups = 3 * nlist;
    k_pme_prep<<<(groups + 7) / 8, 128, 0, st>>>(d_frac, d_list, nlist, order, geo, base, M);
    OFDFT_LAUNCH_CHECK();
    auto tiles = [](int n) { return (n + kPmeTile - 1) / kPmeTile; };
    const unsigned nt = (unsigned)tiles(geo.n0) * tiles(geo.n1) * ((geo.n2 + kPmeTile * kPmeLong - 1) / (kPmeTile * kPmeLong));
    int *counts = nullptr, *starts = nullptr, *lists = nullptr;
    if (nlist >= kPmeSlabAtoms) {
        const int slabs = tiles(geo.n0);
        const long long room = (long long)nlist * std::min(slabs, pme_slabs_of(order));
        counts = (int*)sc.get(prefix + "slabs", 2 * (size_t)slabs * sizeof(int));
        starts = counts + slabs;
        lists = (int*)sc.get(prefix + "lists", (size_t)room * sizeof(int));
        k_pme_slabs<false><<<slabs, kPmeThreads, 0, st>>>(nlist, order, base, geo.n0, counts, starts, lists, room);
        OFDFT_LAUNCH_CHECK();
        k_pme_slabs<true><<<slabs, kPmeThreads, 0, st>>>(nlist, order, base, geo.n0, counts, starts, lists, room);
        OFDFT_LAUNCH_CHECK();
    }
    k_pme_tiles<T><<<nt, kPmeThreads, 0, st>>>(nlist, order, base, M, d_w, d_list, geo, Q, counts, starts, lists);
    OFDFT_LAUNCH_CHECK();
}

// One block per atom: g_a = sum_{ijk} (dQ/du . cinv) * field[l(ijk)], the PME
// gradient of _ForcePME / Forces_rec_PME with dQ_d = n_d dM_d (M_{order-1}
// differences) times the other two M_order factors.  out[3a+c] = scale_a * g_c.
// A thread takes the k2 row of one (i, j): sums of the row with M2 and with dM2 (two
// operations per point), then its three products.
constexpr int kGatherThreads = 128;
template <typename T>
__global__ void __launch_bounds__(kGatherThreads)
    k_pme_gather(const double* __restrict__ frac, const int* __restrict__ sel, int order, Geo geo,
                 const T* __restrict__ field, const double* __restrict__ cinv, const double* __restrict__ scale,
                 double* out) {
    __shared__ double M[3][kMaxOrder];
    __shared__ double dM[3][kMaxOrder];
    __shared__ int at[3][kMaxOrder];
    __shared__ double red[3][kGatherThreads / 32];
    const int a = sel ? sel[blockIdx.x] : blockIdx.x;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (threadIdx.x < 64) {  // two whole warps: the fourth group of 16 repeats an axis
        const int d = (int)(threadIdx.x >> 4) % 3, n = (threadIdx.x & 15) + 1;
        const int nr = d == 0 ? geo.n0 : (d == 1 ? geo.n1 : geo.n2);
        const double up = frac[3 * a + d] * (double)nr, fl = floor(up);
        double before;
        const double v = bspline_mn_lane(up - fl, order, n, before);
        // dM[i] = n_d (M_{order-1}(i+1) - M_{order-1}(i)), M_{order-1}(0) = M_{order-1}(order) = 0
        const double mine = n < order ? before : 0.0;
        double below = __shfl_up_sync(0xffffffffu, mine, 1, 16);
        if (n == 1) below = 0.0;
        if (n <= order && threadIdx.x < 48) {
            M[d][n - 1] = v;
            dM[d][n - 1] = (double)nr * (mine - below);
            at[d][n - 1] = pmod(1LL + (long long)fl - (n - 1), nr);
        }
    }
    __syncthreads();
    double g0 = 0.0, g1 = 0.0, g2 = 0.0;
    for (int t = threadIdx.x; t < order * order; t += kGatherThreads) {
        const int i = t / order, j = t - i * order;
        const T* row = field + ((long long)at[0][i] * geo.n1 + at[1][j]) * geo.n2;
        double s = 0.0, e = 0.0;
        for (int k = 0; k < order; ++k) {
            const double f = (double)row[at[2][k]];
            s += M[2][k] * f;
            e += dM[2][k] * f;
        }
        g0 += dM[0][i] * M[1][j] * s;
        g1 += M[0][i] * dM[1][j] * s;
        g2 += M[0][i] * M[1][j] * e;
    }
    for (int o = 16; o > 0; o >>= 1) {
        g0 += __shfl_down_sync(0xffffffffu, g0, o);
        g1 += __shfl_down_sync(0xffffffffu, g1, o);
        g2 += __shfl_down_sync(0xffffffffu, g2, o);
    }
    if (lane == 0) {
        red[0][wid] = g0;
        red[1][wid] = g1;
        red[2][wid] = g2;
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        double s0 = 0, s1 = 0, s2 = 0;
        for (int w = 0; w < kGatherThreads / 32; ++w) {
            s0 += red[0][w];
            s1 += red[1][w];
            s2 += red[2][w];
        }
        // (dQ . cinv)_c = sum_d dQ_d cinv[d][c]
        const int c = threadIdx.x;
        out[3 * a + c] = (scale ? scale[a] : 1.0) * (s0 * cinv[c] + s1 * cinv[3 + c] + s2 * cinv[6 + c]);
    }
}

// One warp per row (i, j) of the half grid, lanes along k: what a row shares is computed
// once per row instead of once per point.
struct HalfRow {
    int i, j;
    double px, py, pz;  // f0 b0 + f1 b1, rounded as gvec rounds it
    double xr, xi;      // bm0(i) bm1(j)
};
__device__ __forceinline__ HalfRow half_row(const Geo& g, int row, const double* bre, const double* bim) {
    HalfRow r;
    r.i = row / g.n1;
    r.j = row - r.i * g.n1;
    const double f0 = __dmul_rn((double)freq_index(r.i, g.n0), g.fv[0]);
    const double f1 = __dmul_rn((double)freq_index(r.j, g.n1), g.fv[1]);
    r.px = __dadd_rn(__dmul_rn(f0, g.b[0]), __dmul_rn(f1, g.b[3]));
    r.py = __dadd_rn(__dmul_rn(f0, g.b[1]), __dmul_rn(f1, g.b[4]));
    r.pz = __dadd_rn(__dmul_rn(f0, g.b[2]), __dmul_rn(f1, g.b[5]));
    r.xr = r.xi = 0.0;
    if (bre) {
        const double ar = bre[r.i], ai = bim[r.i], cr = bre[g.n0 + r.j], ci = bim[g.n0 + r.j];
        r.xr = ar * cr - ai * ci;
        r.xi = ar * ci + ai * cr;
    }
    return r;
}
// |G|^2 of element k of the row, the bits of gsq()
__device__ __forceinline__ double row_gsq(const Geo& g, const HalfRow& r, int k) {
    const double f2 = __dmul_rn((double)k, g.fv[2]);
    const double gx = __dadd_rn(r.px, __dmul_rn(f2, g.b[6]));
    const double gy = __dadd_rn(r.py, __dmul_rn(f2, g.b[7]));
    const double gz = __dadd_rn(r.pz, __dmul_rn(f2, g.b[8]));
    return __dadd_rn(__dadd_rn(__dmul_rn(gx, gx), __dmul_rn(gy, gy)), __dmul_rn(gz, gz));
}
__device__ __forceinline__ void row_barray(const Geo& g, const HalfRow& r, const double* bre, const double* bim, int k,
                                           double& br, double& bi) {
    const double er = bre[g.n0 + g.n1 + k], ei = bim[g.n0 + g.n1 + k];
    br = r.xr * er - r.xi * ei;
    bi = r.xr * ei + r.xi * er;
}
constexpr int kRowWarps = 8;  // warps (rows) per block of the row kernels
inline int row_grid(const Geo& g, int sms) {
    return blocks_for((long long)g.n0 * g.n1, kRowWarps, sms * 16);
}

// B(G) = bm0(i) bm1(j) bm2(k) from per-axis complex tables (ewald.py:44-55)
__device__ inline void barray(const double* bre, const double* bim, const Geo& g, long long idx, double& br,
                              double& bi) {
    int i, j, k;
    half_index(g, idx, i, j, k);
    // axis offsets in the packed tables: [0, n0), [n0, n0+n1), [n0+n1, ...)
    double ar = bre[i], ai = bim[i];
    double cr = bre[g.n0 + j], ci = bim[g.n0 + j];
    double xr = ar * cr - ai * ci, xi = ar * ci + ai * cr;
    double er = bre[g.n0 + g.n1 + k], ei = bim[g.n0 + g.n1 + k];
    br = xr * er - xi * ei;
    bi = xr * ei + xi * er;
}

}  // namespace ofdft
