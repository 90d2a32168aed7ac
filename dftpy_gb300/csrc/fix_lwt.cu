// The density-dependent (k_F-node) kernel in float64 on integer-pipe transforms (fix_fft.cuh,
// fix_3d.cuh): the quantities of the general path's k_lwt_nodes / interp / pot2 (total.cu;
// lwt.py:226-306), arranged as the float32 fused pipeline is:
//   C2R: k_fx_nodes   K_j and K'_j/k_j times FFT(rho^beta)/N, axis 0 inverse, per node
//        k_fx_axis1   axis 1 inverse, rows that a node needs
//        k_fx_rows    axis 2 C2R, interpolated into pot1 / pot3 at the points of the row
//   R2C: k_fx_hats    hat weights times rho^alpha, axis 2 R2C
//        k_fx_axis1   axis 1 forward
//        k_fx_pot2    axis 0 forward, times K_j (K'_j/k_j) / N, summed into pot2(G)
// A point takes part in the two nodes of its interval only, so rows that no point ties to a
// node are left out, and a plane's value is converted back to float64 at about 1 in 30 points.
//
// 64 x 72 x 80 with 64 nodes (linear, potential): 8.8 ms an evaluation on float64 library
// transforms, 2.9 ms here, of which nodes 0.66, axis 1 0.38 + 0.22, rows 0.43, pot2 0.36,
// hats 0.22 ms and the local terms 0.5 (profiles/fix_kernels_float64.md).
#include "fix_eval.h"

#include "fix_3d.cuh"

#include <algorithm>
#include <vector>

using namespace ofdft;
using namespace ofdft::fix;

namespace {

// ---- kernel table
struct TabK {
    const double* c;   // K: four coefficients per interval
    const double* cd;  // -eta K'
    const double* x;   // l step
    int nint;
    float inv_step, below;  // below: under etamax by more than float32 rounding
    double etamax, limit, limitd;
};

// A positive double within float32's normal range, truncated; on the integer pipe
__device__ __forceinline__ float low_bits_off(double v) {
    const int hi = __double2hiint(v);
    return __int_as_float((int)__funnelshift_l((unsigned)__double2loint(v), (unsigned)hi, 3) - (896 << 23));
}
// K (deriv false) or -eta K' at eta = q ik (fk: ik in float32).  The interval comes from
// float32: at a knot the neighbouring piece, continued over a rounding error, has the same value.
__device__ __forceinline__ double table_at(const TabK& t, bool deriv, double q, double ik, float fk) {
    const float eta = low_bits_off(q) * fk;
    if (!(eta < t.below) && !(q * ik < t.etamax)) return deriv ? t.limitd : t.limit;
    const int l = min(max((int)(eta * t.inv_step), 0), t.nint - 1);
    const double2* p = reinterpret_cast<const double2*>(deriv ? t.cd : t.c) + 2 * (long long)l;
    const double2 a = __ldg(p), b = __ldg(p + 1);
    const double u = fma(q, ik, -__ldg(t.x + l));
    return fma(fma(fma(b.y, u, b.x), u, a.y), u, a.x);
}

// ---- intervals
// il: the last interval (k_i, k_{i+1} + 1e-18) that holds kf, -1 none, -2 the small-k_F branch;
// two: interval il - 1 holds it as well (lwt.py:252-306)
struct Place {
    int il;
    bool two;
};
__device__ __forceinline__ Place place_of(double kf, const double* kn, const double* kup, int m) {
    int lo = 0, hi = m;  // nodes strictly below kf
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (kn[mid] < kf) lo = mid + 1;
        else hi = mid;
    }
    auto in = [&](int i) { return i >= 0 && i <= m - 2 && kf < kup[i + 1]; };
    Place p;
    p.two = false;
    if (in(lo - 1)) {
        p.il = lo - 1;
        p.two = in(lo - 2);
    } else if (in(lo - 2)) {
        p.il = lo - 2;
    } else {
        p.il = kf < kup[0] ? -2 : -1;
    }
    return p;
}

struct Lwt {
    Grid3 g;
    Geo geo;
    TabK tab;
    const double* kf;
    const double* rA;
    const double2* rbG;
    double *p1[4], *p3[4];  // pot1, pot3 from the lower and upper nodes' P, M planes; null: no part
    double2* pot2G;
    double2* XY;        // planes: P then M (C2R), hats (R2C)
    long long plane;
    const double* kn;
    const double* invk;
    const double* kup;
    const unsigned* need;  // bit i1 % 32 of [(i0 m + j) words + i1 / 32]
    const short* code;     // per point: 2 il + two (Place)
    const double* t;       // and its interval coordinate (small branch: (kf - k_0) / k_0)
    int m, words, j0, nb, nm;  // nm: planes per node of the chain (1 or 2)
    int lb, lines, share, first, hermite;
    FastDiv dn, dh;
    double kfclip, invN;
};

__device__ __forceinline__ bool needed(const Lwt& a, int i0, int i1, int j) {
    return (__ldg(a.need + ((long long)i0 * a.m + j) * a.words + (i1 >> 5)) >> (i1 & 31)) & 1u;
}

// Interval and coordinate of every point, and the need bits of 32 rows (one i0, one word of i1)
// collected in shared memory
__global__ void __launch_bounds__(1024) k_fx_need(Lwt a, unsigned* __restrict__ out, short* __restrict__ code,
                                                 double* __restrict__ t) {
    extern __shared__ double need_sm[];
    double* kn = need_sm;
    double* kup = kn + a.m;
    unsigned* bits = reinterpret_cast<unsigned*>(kup + a.m);
    const int i0 = blockIdx.x / a.words, word = blockIdx.x % a.words;
    for (int q = threadIdx.x; q < a.m; q += blockDim.x) {
        kn[q] = a.kn[q];
        kup[q] = a.kup[q];
        bits[q] = 0;
    }
    __syncthreads();
    const int n1 = a.g.n1, n2 = a.g.n2, lane = threadIdx.x & 31;
    for (int r = threadIdx.x >> 5; r < 32; r += (int)blockDim.x >> 5) {
        const int i1 = word * 32 + r;
        if (i1 >= n1) break;
        const long long row = ((long long)i0 * n1 + i1) * n2;
        int last = -3;
        for (int i = lane; i < n2; i += 32) {
            const double kf = fmin(a.kf[row + i], a.kfclip);
            const Place p = place_of(kf, kn, kup, a.m);
            const int at = max(p.il, 0);
            code[row + i] = (short)(2 * p.il + p.two);
            t[row + i] = (kf - kn[at]) / (p.il >= 0 ? kn[at + 1] - kn[at] : kn[0]);
            if (p.il == last && !p.two) continue;
            last = p.il;
            const int lo = p.il == -2 ? 0 : p.il - p.two, hi = p.il == -2 ? 0 : p.il + 1;
            if (p.il != -1)
                for (int j = lo; j <= hi; ++j) atomicOr(bits + j, 1u << r);
        }
    }
    __syncthreads();
    for (int q = threadIdx.x; q < a.m; q += blockDim.x) out[((long long)i0 * a.m + q) * a.words + word] = bits[q];
}

// |G| of the elements of a column tile of axis 0 and FFT(rho^beta)/N there (z may be null)
__device__ __forceinline__ void stage_column(const Lwt& a, int lb, double* sq, double2* sz) {
    const int L = 1 << lb, n = a.g.n0, l = threadIdx.x & (L - 1);
    const int line = (blockIdx.x % a.lines << lb) + l;
    const bool in = line < col_lines<0>(a.g);
    const int k1 = line / a.g.n2h, k2 = line - k1 * a.g.n2h;
    const long long stride = col_stride<0>(a.g);
    for (int i = threadIdx.x >> lb; i < n; i += blockDim.x >> lb) {
        const long long at = line + i * stride;
        sq[i * (L + 1) + l] = in && at != 0 ? sqrt(gsq(a.geo, at)) : 1.0;  // K_j(0) = 0: any value will do
        if (sz) {
            double2 z = make_double2(0.0, 0.0);
            if (in && at != 0) {  // K_j(0) = 0
                z = a.rbG[at];
                z.x *= a.invN;
                z.y *= a.invN;
            }
            sz[i * (L + 1) + l] = z;
        }
    }
    __syncthreads();
}

// Axis 0 inverse of K_j FFT(rho^beta)/N (plane jj) and, nm = 2, K'_j/k_j FFT(rho^beta)/N (plane
// nb + jj) for the block's share of the batch's nodes; |G| and FFT(rho^beta)/N of the tile stay
// in shared memory.  Bound by the float64 pipe, 82% busy at 64 x 72 x 80: eleven operations per
// value (table 4, product 2, conversions 5); the interval's float32 argument is taken from the
// bits instead of converted, and K'_j's factor 1/k_j is left to the points that use it.
__global__ void __launch_bounds__(kThreads, kBlocks) k_fx_nodes(Lwt a) {
    extern __shared__ __align__(16) unsigned char fix_smem[];
    __shared__ LineSm sm;
    const Plan& p = a.g.p0;
    const int n = p.n, lb = a.lb, L = 1 << lb, LP = L + 1;
    I2* b0 = reinterpret_cast<I2*>(fix_smem);
    I2* b1 = b0 + (p.np == 3 ? n * LP : 0);
    double2* sz = reinterpret_cast<double2*>(b1 + n * LP);
    double* sq = reinterpret_cast<double*>(sz + n * LP);
    stage_column(a, lb, sq, sz);
    const int tile = blockIdx.x % a.lines, part = blockIdx.x / a.lines;
    const int line = (tile << lb) + (threadIdx.x & (L - 1));
    const bool in = line < col_lines<0>(a.g);
    const long long stride = col_stride<0>(a.g);
    const int s1 = min(a.nb, (part + 1) * a.share);
    for (int jj = part * a.share; jj < s1; ++jj) {
        const double ik = a.invk[a.j0 + jj];
        const float fk = (float)ik;
        for (int d = 0; d < a.nm; ++d) {
            double2* base = a.XY + (long long)(d * a.nb + jj) * a.plane + (in ? line : 0);
            tile_fft_out(
                b0, b1, p, lb, sm,
                [&](int i, int l) {
                    const double K = table_at(a.tab, d != 0, sq[i * LP + l], ik, fk);
                    const double2 z = sz[i * LP + l];
                    return make_double2(z.y * K, z.x * K);  // parts exchanged: the inverse
                },
                [&](int i, int l, I2 z) {
                    if (in) __stcs(base + i * stride, swapped(from_fix(z, sm, l)));
                });
            __syncthreads();  // the scales are read before the next transform resets them
        }
    }
}

// Axis 1 of the planes (node j0 + plane % nb), in place: the inverse stores and the forward
// transform reads the rows that the node needs only.  Issue slots 49% used with the 14 warps per
// SM that the registers allow (ALU 44%, float64 34%).
template <bool INV>
__global__ void __launch_bounds__(kThreads, kBlocks) k_fx_axis1(Lwt a) {
    extern __shared__ __align__(16) unsigned char fix_smem[];
    __shared__ LineSm sm;
    const Plan& p = a.g.p1;
    I2* b0 = reinterpret_cast<I2*>(fix_smem);
    const int line = (blockIdx.x << a.lb) + (threadIdx.x & ((1 << a.lb) - 1));
    const bool in = line < col_lines<1>(a.g);
    const int j = a.j0 + blockIdx.y % a.nb, i0 = in ? line / a.g.n2h : 0, h = a.g.n2h;
    double2* base = a.XY + (long long)blockIdx.y * a.plane + (in ? col_base<1>(a.g, line) : 0);
    const unsigned* bits = a.need + ((long long)i0 * a.m + j) * a.words;
    auto on = [&](int i) { return (__ldg(bits + (i >> 5)) >> (i & 31)) & 1u; };
    tile_fft_out(
        b0, b0 + p.n * ((1 << a.lb) + 1), p, a.lb, sm,
        [&](int i, int) {
            if (!in || (!INV && !on(i))) return make_double2(0.0, 0.0);
            const double2 v = base[(long long)i * h];
            return INV ? swapped(v) : v;
        },
        [&](int i, int l, I2 z) {
            if (!in || (INV && !on(i))) return;
            const double2 v = from_fix(z, sm, l);
            base[(long long)i * h] = INV ? swapped(v) : v;
        });
}

// The row passes: a block has two rows (one complex line) and transforms them for its part of
// the planes that they need, as many at a time as the tile has lines.  One row pair per tile keeps the
// list short (a warp with eight rows to a node transformed 1.5 times as much), and warps that
// run the same passes together share the instruction cache (fetches are still the most common
// stall of k_fx_rows).  In shared memory: the codes of the points and the planes' list (2 node + plane).
struct RowPair {
    long long row0;
    int two;                // rows: 1 or 2
    short2* code;           // of point i in both rows
    unsigned short* list;
    unsigned char* both;    // rows that need the plane: 1, 2 or both
    int from, to;           // the block's part of the list (blockIdx.y), whole tiles
};
__device__ __forceinline__ RowPair stage_rows(const Lwt& a, void* at, int* counter) {
    RowPair s;
    const int n = a.g.n2, n1 = a.g.n1, T = blockDim.x;
    s.row0 = 2LL * blockIdx.x;
    s.two = min(2LL, (long long)a.g.n0 * n1 - s.row0);
    s.code = reinterpret_cast<short2*>(at);
    s.list = reinterpret_cast<unsigned short*>(s.code + n);
    s.both = reinterpret_cast<unsigned char*>(s.list + a.nb * a.nm);
    if (threadIdx.x < 32) {  // in order
        const int i0 = (int)s.row0 / n1, i1 = (int)s.row0 - i0 * n1;
        const int k1 = i1 + 1 == n1 ? 0 : i1 + 1, k0 = i0 + (k1 == 0);
        int c = 0;
        for (int q0 = 0; q0 < a.nb; q0 += 32) {
            const int q = q0 + threadIdx.x;
            int on = 0;
            if (q < a.nb) {
                on = needed(a, i0, i1, a.j0 + q);
                if (s.two == 2) on |= 2 * needed(a, k0, k1, a.j0 + q);
            }
            const unsigned all = __ballot_sync(~0u, on != 0);
            if (on) {
                const int k = a.nm * (c + __popc(all & ((1u << threadIdx.x) - 1u)));
                for (int d = 0; d < a.nm; ++d) {
                    s.list[k + d] = (unsigned short)(2 * q + d);
                    s.both[k + d] = (unsigned char)on;
                }
            }
            c += __popc(all);
        }
        if (threadIdx.x == 0) *counter = c * a.nm;
    }
    for (int i = threadIdx.x; i < n; i += T)
        s.code[i] = make_short2(a.code[s.row0 * n + i], s.two == 2 ? a.code[(s.row0 + 1) * n + i] : (short)-2);
    __syncthreads();
    const int c = *counter, per = (((c + (1 << a.lb) - 1) >> a.lb) + gridDim.y - 1) / gridDim.y << a.lb;
    s.from = min(c, (int)blockIdx.y * per);
    s.to = min(c, s.from + per);
    return s;
}
inline size_t rows_smem(int n, int planes) { return (size_t)n * sizeof(short2) + (size_t)planes * 3 + 16; }

// Weights of node j at a point of interval i (t its coordinate, D its width): j = i (lo) or
// j = i + 1; for the P plane w1 (pot1) and w3 (pot3), for the M plane m1 and m3
struct Weights {
    double w1, w3, m1, m3;
};
__device__ __forceinline__ Weights weights(bool hermite, bool lo, double t, double D) {
    if (!hermite) {
        const double w = lo ? 1.0 - t : t;
        return Weights{w, 0.0, 0.0, w};
    }
    const double t2 = t * t, t3 = t2 * t, h00 = 2.0 * t3 - 3.0 * t2 + 1.0, d = (6.0 * t2 - 6.0 * t) / D;
    if (lo) return Weights{h00, d, D * (t3 - 2.0 * t2 + t), 3.0 * t2 - 4.0 * t + 1.0};
    return Weights{1.0 - h00, -d, D * (t3 - t2), 3.0 * t2 - 2.0 * t};
}

// Axis 2 C2R, interpolated where a point's interval ends at the plane's node.  Each plane has
// its own part of pot1 and pot3 at a point, so nothing is summed between threads.
__global__ void __launch_bounds__(kThreads, kBlocks) k_fx_rows(Lwt a) {
    extern __shared__ __align__(16) unsigned char fix_smem[];
    __shared__ LineSm sm;
    __shared__ int count;
    const Plan& p = a.g.p2;
    const int n = p.n, h = a.g.n2h, L = 1 << a.lb, LP = L + 1, T = blockDim.x;
    I2* b0 = reinterpret_cast<I2*>(fix_smem);
    I2* b1 = b0 + (p.np == 3 ? n * LP : 0);
    const RowPair s = stage_rows(a, b1 + n * LP, &count);
    if (a.first && blockIdx.y == 0) {  // ends that no plane writes
        for (int e = threadIdx.x; e < s.two * n; e += T) {
            const int i = a.dn.div(e) ? e - n : e, cd = e < n ? s.code[i].x : s.code[i].y;
            if (cd >= 0) continue;
            for (int k = 0; k < 4; ++k) {
                if (a.p1[k] && !(cd == -4 && k == 0)) a.p1[k][s.row0 * n + e] = 0.0;
                if (a.p3[k]) a.p3[k][s.row0 * n + e] = 0.0;
            }
        }
    }
    double2* raw = reinterpret_cast<double2*>(b0);
    for (int q0 = s.from; q0 < s.to; q0 += L) {
        __syncthreads();  // the buffer and the scales are free
        for (int e = threadIdx.x; e < L * h; e += T) {
            const int l = a.dh.div(e), k = e - l * h, q = q0 + l;
            double2 A = make_double2(0.0, 0.0), B = A;
            if (q < s.to) {
                const int it = s.list[q], on = s.both[q];  // a row that the node does not need holds no values
                const double2* in = a.XY + (long long)((it & 1) * a.nb + (it >> 1)) * a.plane + s.row0 * h + k;
                if (on & 1) A = __ldcs(in);
                if (on & 2) B = __ldcs(in + h);
            }
            join_rows(raw, A, B, k, l, n, LP);
        }
        __syncthreads();
        tile_fft_out(
            b0, b1, p, a.lb, sm, [&](int i, int l) { return raw[i * LP + l]; },
            [&](int i, int l, I2 v) {
                if (q0 + l >= s.to) return;
                const int it = s.list[q0 + l], j = a.j0 + (it >> 1), d = it & 1;
                const short2 two = s.code[i];
                for (int b = 0; b < 2; ++b) {
                    const int cd = b ? two.y : two.x, il = cd >> 1;
                    const bool small = cd == -4 && j == 0 && d == 0, in_lo = cd >= 0 && il == j;
                    if (!(small || in_lo || (cd >= 0 && il == j - 1))) continue;
                    const long long o = (s.row0 + b) * n + i;
                    double f = to_dbl(b ? v.x : v.y, sm.ds[l] - sm.k[l], sm.emax[l] == kNonFinite);
                    const double t = a.t[o];
                    if (small) {
                        a.p1[0][o] = f * t;
                        continue;
                    }
                    if (d) f *= a.invk[j];
                    const Weights w = weights(a.hermite, in_lo, t, a.hermite ? a.kn[il + 1] - a.kn[il] : 0.0);
                    const int k = (in_lo ? 0 : 2) + d;
                    if (a.p1[k]) a.p1[k][o] = (d ? w.m1 : w.w1) * f;
                    if (a.p3[k]) a.p3[k][o] = (d ? w.m3 : w.w3) * f;
                }
            });
    }
}

// rho^alpha times the hat weights of the needed nodes (plane jj; Hermite: and the derivative
// weights, which take K'_j's 1/k_j, plane nb + jj), axis 2 R2C
__global__ void __launch_bounds__(kThreads, kBlocks) k_fx_hats(Lwt a) {
    extern __shared__ __align__(16) unsigned char fix_smem[];
    __shared__ LineSm sm;
    __shared__ int count;
    const Plan& p = a.g.p2;
    const int n = p.n, h = a.g.n2h, L = 1 << a.lb, LP = L + 1, T = blockDim.x;
    I2* b0 = reinterpret_cast<I2*>(fix_smem);
    I2* b1 = b0 + n * LP;
    const RowPair s = stage_rows(a, b1 + n * LP, &count);
    for (int q0 = s.from; q0 < s.to; q0 += L) {
        auto hat = [&](int cd, int j, int d, long long o) {
            const int il = cd >> 1;
            const bool small = cd == -4 && j == 0 && d == 0, here = cd >= 0 && (il == j || il == j - 1);
            const bool below = cd > 0 && (cd & 1) && (il == j || il - 1 == j);  // the interval below holds it too
            if (!(small || here || below)) return 0.0;
            const double t = a.t[o];
            if (small) return a.rA[o] * t;
            const double D = a.kn[il + 1] - a.kn[il];
            double w = 0.0;
            if (here) {
                const Weights x = weights(a.hermite, il == j, t, D);
                w = d ? x.m1 : x.w1;
            }
            if (below) {
                const double E = a.kn[il] - a.kn[il - 1];
                const Weights x = weights(a.hermite, il - 1 == j, (E + t * D) / E, E);
                w += d ? x.m1 : x.w1;
            }
            return a.rA[o] * (d ? w * a.invk[j] : w);
        };
        __syncthreads();  // the buffers and the scales are free
        const I2* z = tile_fft(b0, b1, p, a.lb, sm, [&](int i, int l) {
            double2 v = make_double2(0.0, 0.0);
            if (q0 + l < s.to) {
                const int it = s.list[q0 + l], j = a.j0 + (it >> 1), d = it & 1;
                const short2 two = s.code[i];
                v.x = hat(two.x, j, d, s.row0 * n + i);
                v.y = hat(two.y, j, d, (s.row0 + 1) * n + i);
            }
            return v;
        });
        for (int e = threadIdx.x; e < L * h; e += T) {
            const int l = a.dh.div(e), k = e - l * h, q = q0 + l;
            if (q >= s.to) break;
            const int it = s.list[q], on = s.both[q];
            const I2 Z = z[k * LP + l], Y = z[(k ? n - k : 0) * LP + l];
            double2* out = a.XY + (long long)((it & 1) * a.nb + (it >> 1)) * a.plane + s.row0 * h + k;
            if (on & 1) __stcs(out, from_fix(I2{Z.x + Y.x, Z.y - Y.y}, sm, l, -1));
            if (on & 2) __stcs(out + h, from_fix(I2{Z.y + Y.y, Y.x - Z.x}, sm, l, -1));
        }
    }
}

// Axis 0 forward of the hat planes, times K_j (plane jj) or K'_j/k_j (plane nb + jj) over N,
// summed over the block's share of the nodes into pot2(G) (share = nb) or into one partial
// spectrum per share.  Float64 pipe 82% busy, as k_fx_nodes.
__global__ void __launch_bounds__(kThreads, kBlocks) k_fx_pot2(Lwt a) {
    extern __shared__ __align__(16) unsigned char fix_smem[];
    __shared__ LineSm sm;
    const Plan& p = a.g.p0;
    const int n = p.n, lb = a.lb, L = 1 << lb, LP = L + 1;
    I2* b0 = reinterpret_cast<I2*>(fix_smem);
    I2* b1 = b0 + (p.np == 3 ? n * LP : 0);
    double2* acc = reinterpret_cast<double2*>(b1 + n * LP);
    double* sq = reinterpret_cast<double*>(acc + n * LP);
    stage_column(a, lb, sq, nullptr);
    const int tile = blockIdx.x % a.lines, part = blockIdx.x / a.lines, l = threadIdx.x & (L - 1);
    const int line = (tile << lb) + l;
    const bool in = line < col_lines<0>(a.g);
    const long long stride = col_stride<0>(a.g);
    for (int i = threadIdx.x >> lb; i < n; i += blockDim.x >> lb) acc[i * LP + l] = make_double2(0.0, 0.0);
    const int s1 = min(a.nb, (part + 1) * a.share);
    for (int jj = part * a.share; jj < s1; ++jj) {
        const double ik = a.invk[a.j0 + jj];
        const float fk = (float)ik;
        for (int d = 0; d < a.nm; ++d) {
            const double2* base = a.XY + (long long)(d * a.nb + jj) * a.plane + (in ? line : 0);
            tile_fft_out(
                b0, b1, p, lb, sm, [&](int i, int) { return in ? __ldcs(base + i * stride) : make_double2(0.0, 0.0); },
                [&](int i, int q, I2 z) {
                    const double K = table_at(a.tab, d != 0, sq[i * LP + q], ik, fk);
                    const double2 v = from_fix(z, sm, q);
                    double2 t = acc[i * LP + q];
                    t.x = fma(K, v.x, t.x);
                    t.y = fma(K, v.y, t.y);
                    acc[i * LP + q] = t;
                });
            __syncthreads();  // the scales are read before the next transform resets them
        }
    }
    if (!in) return;
    double2* out = a.pot2G + (long long)part * a.plane + line;
    for (int i = threadIdx.x >> lb; i < n; i += blockDim.x >> lb) {
        double2 t = acc[i * LP + l];
        t.x *= a.invN;
        t.y *= a.invN;
        if (i == 0 && line == 0) t = make_double2(0.0, 0.0);  // K_j(0) = 0
        const double2 old = a.first ? make_double2(0.0, 0.0) : out[i * stride];
        out[i * stride] = make_double2(old.x + t.x, old.y + t.y);
    }
}

// the partial spectra, in order, into the first
__global__ void k_fx_join(double2* __restrict__ x, long long n, int parts) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        double2 s = x[i];
        for (int k = 1; k < parts; ++k) {
            const double2 v = x[(long long)k * n + i];
            s.x += v.x;
            s.y += v.y;
        }
        x[i] = s;
    }
}

// blocks per SM of a kernel of 128 registers
int resident(int threads, size_t smem) {
    return (int)std::max<size_t>(1, std::min((size_t)(kThreads * kBlocks / threads), (size_t)(227 * 1024) / (smem + 1500)));
}
// Into how many shares the nodes are split over `tiles` blocks each: the fewest rounds of
// resident blocks, a block costing its nodes and one more for its start
int shares(int nodes, int most, long long tiles, long long slots) {
    int best = 1;
    double cost = 1e300;
    for (int s = 1; s <= std::min(nodes, most); ++s) {
        const double c = (double)((tiles * s + slots - 1) / slots) * ((nodes + s - 1) / s + 1);
        if (c < 0.98 * cost) {
            cost = c;
            best = s;
        }
    }
    return best;
}

// lines per tile of a kernel that keeps more than the transform in shared memory
Shape fit(const Plan& p, long long lines, int sms, size_t per_line) {
    Shape s = shape_of(p, lines, sms);
    while (s.lb > 0 && tile_smem(p, s.lb, 1) + per_line * ((1 << s.lb) + 1) > 56 * 1024) {
        --s.lb;
        s.threads = (((p.n / p.r[0]) << s.lb) + 31) / 32 * 32;
    }
    return s;
}

}  // namespace

namespace ofdft {
namespace fix {

int lwt_enqueue(ofdft_grid* g, Scratch& sc, const LwtArgs& r, cudaStream_t st) {
    const Grid3& p = *grid_plans(g);
    const int sms = g->sms;
    const size_t cb = g->cplx_bytes();
    Lwt a{};
    a.g = p;
    a.geo = g->geo;
    a.tab = TabK{r.tab_c, r.tab_cd, r.tab_x, r.nint, (float)(1.0 / r.step), (float)(r.etamax * (1.0 - 1e-6)), r.etamax, r.limit, r.limitd};
    a.kf = r.kf;
    a.rA = r.rA;
    a.rbG = r.rbG;
    for (int i = 0; i < 4; ++i) {
        a.p1[i] = r.pot1[i];
        a.p3[i] = r.pot3[i];
    }
    a.plane = g->Nc;
    a.kn = r.kn;
    a.invk = r.invk;
    a.kup = r.kup;
    a.m = r.m;
    a.words = (p.n1 + 31) / 32;
    a.hermite = r.hermite;
    a.kfclip = r.kfclip;
    a.invN = 1.0 / (double)g->N;
    a.dn = fast_div(p.n2);
    a.dh = fast_div(p.n2h);
    int launches = 0;

    unsigned* need = (unsigned*)sc.get("fx_need", (size_t)p.n0 * r.m * a.words * sizeof(unsigned));
    short* code = (short*)sc.get("fx_code", (size_t)g->N * sizeof(short));
    double* t = (double*)sc.get("fx_t", g->real_bytes());
    a.need = need;
    a.code = code;
    a.t = t;
    double share = 1.0;  // of the rows that are needed: for the byte counts of a timed run
    {
        const size_t smem = (size_t)r.m * (2 * sizeof(double) + sizeof(unsigned));
        smem_optin(k_fx_need, smem);
        r.time(INTERP, (double)g->N * (2 * sizeof(double) + sizeof(short)), st, [&] {
            k_fx_need<<<p.n0 * a.words, std::min(32, p.n1) * 32, smem, st>>>(a, need, code, t);
        });
        ++launches;
        if (r.time.owner) {
            std::vector<unsigned> bits((size_t)p.n0 * r.m * a.words);
            OFDFT_CK(cudaMemcpyAsync(bits.data(), need, bits.size() * sizeof(unsigned), cudaMemcpyDeviceToHost, st));
            OFDFT_CK(cudaStreamSynchronize(st));
            long long on = 0;
            for (unsigned b : bits) on += __builtin_popcount(b);
            share = (double)on / ((double)p.n0 * p.n1 * r.m);
        }
    }
    const double cplx = (double)cb, real = (double)g->real_bytes();
    const bool mc = r.kdd == 3 || r.hermite, hats = r.kdd > 1;
    const int nc = mc ? 2 : 1, nh = hats ? (r.hermite ? 2 : 1) : 0;
    size_t freeb = 0, totalb = 0;
    cudaMemGetInfo(&freeb, &totalb);
    int B = r.max_batch > 0 ? r.max_batch : 64;
    const long long per_node = (long long)(nc + nh) * cb, fits = (long long)(0.5 * (double)freeb) / per_node;
    B = std::min(std::min(B, r.m), (int)std::max(1LL, std::min(fits, 65535LL / 2)));
    double2* XY = (double2*)sc.get("lwtXY", (size_t)nc * B * cb);
    double2* U = hats ? (double2*)sc.get("lwtXY2", (size_t)nh * B * cb) : nullptr;

    // axis-0 passes: |G| (and FFT(rho^beta)/N or the sums) beside the transform
    const Shape s0 = fit(p.p0, col_lines<0>(p), sms, (size_t)p.n0 * (sizeof(double2) + sizeof(double)));
    const int tiles0 = (int)col_blocks(col_lines<0>(p), s0.lb);
    const size_t smem0 = tile_smem(p.p0, s0.lb, 1) + (size_t)p.n0 * ((1 << s0.lb) + 1) * (sizeof(double2) + sizeof(double));
    const long long slots0 = (long long)sms * resident(s0.threads, smem0);
    // k_fx_pot2's shares are partial spectra, so few; k_fx_nodes sums nothing, and splits further
    // where eight shares leave the chip idle
    const int parts = shares(B, 8, tiles0, slots0), nparts = 8 * tiles0 < slots0 ? shares(B, B, tiles0, slots0) : parts;
    const Shape s1 = shape_of(p.p1, col_lines<1>(p), sms);
    const size_t smem1 = tile_smem(p.p1, s1.lb, 1);
    const Shape s2 = shape_of(p.p2, 1LL << 40, sms);
    const size_t smemr = tile_smem(p.p2, s2.lb, 1) + rows_smem(p.n2, nc * B);
    const size_t smemh = tile_smem(p.p2, s2.lb, 2) + rows_smem(p.n2, std::max(nh, 1) * B);
    const unsigned b2 = (unsigned)(((long long)p.n0 * p.n1 + 1) / 2);
    // Row pairs times parts of their planes' lists: as many parts as fill the chip once.  With a
    // block per row pair a grid of few rows waited for lists of up to 128 planes: 64 nodes,
    // Hermite, whole call: 16^3 789 us (568 in parts; general path 650), 4 x 4 x 512 2082 (456; 740),
    // 32^3 792 (764; 1245), 64 x 72 x 80 in one part either way.
    auto row_parts = [&](int planes, size_t smem) {
        const long long slots = (long long)sms * resident(s2.threads, smem), tiles = (planes + (1 << s2.lb) - 1) >> s2.lb;
        return (unsigned)std::max(1LL, std::min(tiles, slots / b2));
    };
    double2* pot2 = hats ? (double2*)sc.get("fx_pot2", (size_t)parts * cb) : nullptr;
    smem_optin(k_fx_nodes, smem0);
    smem_optin(k_fx_pot2, smem0);
    smem_optin(k_fx_axis1<true>, smem1);
    smem_optin(k_fx_axis1<false>, smem1);
    smem_optin(k_fx_rows, smemr);
    smem_optin(k_fx_hats, smemh);
    for (int j0 = 0; j0 < r.m; j0 += B) {
        a.j0 = j0;
        a.nb = std::min(B, r.m - j0);
        a.first = j0 == 0;
        a.XY = XY;
        a.nm = nc;
        a.lb = s0.lb;
        a.lines = tiles0;
        a.share = (a.nb + nparts - 1) / nparts;
        r.time(NODES, cplx * (1 + nc * a.nb), st, [&] {
            k_fx_nodes<<<tiles0 * ((a.nb + a.share - 1) / a.share), s0.threads, smem0, st>>>(a);
        });
        a.lb = s1.lb;
        const unsigned b1 = col_blocks(col_lines<1>(p), s1.lb);
        r.time(AXIS1, cplx * nc * a.nb * (1 + share), st, [&] {
            k_fx_axis1<true><<<dim3(b1, nc * a.nb), s1.threads, smem1, st>>>(a);
        });
        a.lb = s2.lb;
        r.time(INTERP, cplx * nc * a.nb * share + real * 2, st, [&] {
            k_fx_rows<<<dim3(b2, row_parts(nc * a.nb, smemr)), s2.threads, smemr, st>>>(a);
        });
        launches += 3;
        if (!hats) continue;
        a.XY = U;
        a.nm = nh;
        r.time(HATS, cplx * nh * a.nb * share + real * 2, st, [&] {
            k_fx_hats<<<dim3(b2, row_parts(nh * a.nb, smemh)), s2.threads, smemh, st>>>(a);
        });
        a.lb = s1.lb;
        r.time(AXIS1, cplx * nh * a.nb * (1 + share), st, [&] {
            k_fx_axis1<false><<<dim3(b1, nh * a.nb), s1.threads, smem1, st>>>(a);
        });
        a.lb = s0.lb;
        a.pot2G = pot2;
        a.share = (a.nb + parts - 1) / parts;
        const int used = (a.nb + a.share - 1) / a.share;
        if (a.first && used < parts)  // a later, fuller batch may use more partial spectra
            OFDFT_CK(cudaMemsetAsync(pot2 + (size_t)used * g->Nc, 0, (size_t)(parts - used) * cb, st));
        r.time(POT2, cplx * (nh * a.nb + used), st, [&] {
            k_fx_pot2<<<tiles0 * used, s0.threads, smem0, st>>>(a);
        });
        launches += 3;
    }
    if (hats) {
        if (parts > 1) {
            r.time(POT2, cplx * (parts + 1), st, [&] {
                k_fx_join<<<blocks_for(g->Nc, 256, sms * 8), 256, 0, st>>>(pot2, g->Nc, parts);
            });
            ++launches;
        }
        double* out = r.pot2;
        r.time(FFT, 5 * cplx + real, st, [&] { c2r(g, &pot2, &out, 1, st); });
        launches += 3;
    }
    return launches;
}

}  // namespace fix
}  // namespace ofdft
