// Three-dimensional float64 real transforms on the integer pipe (fix_fft.cuh): tiles
// of lines in shared memory, one block per tile, three passes per transform.
//   rows     axis 2: two adjacent rows as one complex line, split into (or joined
//            from) their half spectra
//   columns  axes 1 and 0: tiles of consecutive k2, in place; the axis-0 pass can
//            multiply by a G-space factor and transform back in the same launch
// A launch covers several fields (blockIdx.y), each a half-complex array in cuFFT's
// R2C layout.  The first axis pass of a tile reads its elements straight into the
// registers of its butterflies; the shared buffers hold the exchanges.
#pragma once
#include "common.cuh"
#include "fix_fft.cuh"

namespace ofdft {
namespace fix {

constexpr int kThreads = 128;
constexpr int kMaxFields = 8;

struct Grid3 {
    int n0, n1, n2, n2h;
    Plan p0, p1, p2;
};

// quotient by a divisor known on the host, for dividends below 2^16
struct FastDiv {
    unsigned d, m;
    __device__ __forceinline__ int div(int e) const { return (int)__umulhi((unsigned)e, m); }
};
inline FastDiv fast_div(int d) { return FastDiv{(unsigned)d, (unsigned)(((1ULL << 32) + d - 1) / d)}; }

// What a block keeps of its lines' scales
struct LineSm {
    int emax[8];
    unsigned most[8];  // largest 1-norm of a first-pass subset
    unsigned sum[8];   // 1-norm of the line
    Scale c[8];        // scale during the first pass
    int ds[8];         // shift after it
};

// Lines per tile: the largest power of two up to `most` (at most 8) whose first-pass
// butterflies fit one per thread.
inline int lines_of(const Plan& p, int most) {
    int L = most;
    while (L > 1 && L * (p.n / p.r[0]) > kThreads) L >>= 1;
    return L;
}
inline size_t tile_smem(const Plan& p, int L) { return 2 * (size_t)p.n * (L + 1) * sizeof(I2); }

// First pass: butterfly (j, l) of radix R reads its elements with get(n, l) (float64
// pairs, real and imaginary parts as the transform takes them), agrees on the lines'
// scales and stores its outputs.
template <int R, class Get>
__device__ __forceinline__ void pass0(I2* dst, int n, int lb, LineSm& sm, int np, Get get) {
    const int m = n / R, L = 1 << lb, l = threadIdx.x & (L - 1), j = threadIdx.x >> lb;
    const bool on = j < m;
    double2 v[R];
    int em = 0;
    if (on) {
#pragma unroll
        for (int q = 0; q < R; ++q) {
            v[q] = get(j + q * m, l);
            em = max(em, max(expo(v[q].x), expo(v[q].y)));
        }
        atomicMax(&sm.emax[l], em);
    }
    __syncthreads();
    if (on) {
        em = sm.emax[l];
        unsigned s = 2 * R;
#pragma unroll
        for (int q = 0; q < R; ++q) s += lead(v[q].x, em) + lead(v[q].y, em);
        atomicMax(&sm.most[l], s);
        atomicAdd(&sm.sum[l], s);
    }
    __syncthreads();
    if (on) {
        Scale c;
        c.emax = em;
        c.sh = 32 - __clz((int)sm.most[l]);
        if (j == 0) {
            sm.c[l] = c;
            sm.ds[l] = np > 1 ? (32 - __clz((int)sm.sum[l])) - c.sh : 0;
        }
        I2 u[R];
#pragma unroll
        for (int q = 0; q < R; ++q) u[q] = I2{to_fix(v[q].x, c), to_fix(v[q].y, c)};
        Dft<R>::run(u);
#pragma unroll
        for (int q = 0; q < R; ++q) dst[(j * R + q) * (L + 1) + l] = u[q];
    }
}

// A later pass over the tile, sub-transform length Ns; second: the pass after pass0
template <int R>
__device__ __forceinline__ void pass(const I2* src, I2* dst, int n, int lb, int Ns, const I2* __restrict__ tw,
                                     const LineSm& sm, bool second) {
    const int m = n / R, step = n / (Ns * R), L = 1 << lb;
    for (int it = threadIdx.x; it < m * L; it += kThreads) {
        const int l = it & (L - 1), j = it >> lb, k = j % Ns;
        const int ds = second ? sm.ds[l] : 0;
        I2 u[R];
#pragma unroll
        for (int q = 0; q < R; ++q) {
            u[q] = src[(j + q * m) * (L + 1) + l];
            if (q > 0) {
                const longlong2 w = __ldg(reinterpret_cast<const longlong2*>(tw) + k * q * step);
                u[q] = cmul(u[q], I2{w.x, w.y});
            }
            u[q] = I2{shr(u[q].x, ds), shr(u[q].y, ds)};
        }
        Dft<R>::run(u);
        const int base = (j / Ns) * Ns * R + k;
#pragma unroll
        for (int q = 0; q < R; ++q) dst[(base + q * Ns) * (L + 1) + l] = u[q];
    }
}

#define FIX_RADICES(CASE) \
    CASE(2) CASE(3) CASE(4) CASE(5) CASE(6) CASE(7) CASE(8) CASE(9) CASE(10) CASE(12) CASE(14) CASE(15) CASE(16)

// Transforms the tile's lines; returns the buffer with the result (visible to all).
// Entry: b0 free, no thread still uses sm.
template <class Get>
__device__ __forceinline__ const I2* tile_fft(I2* b0, I2* b1, const Plan& p, int lb, LineSm& sm, Get get) {
    if (threadIdx.x < 8) {
        sm.emax[threadIdx.x] = 0;
        sm.most[threadIdx.x] = 0;
        sm.sum[threadIdx.x] = 0;
    }
    __syncthreads();
    switch (p.r[0]) {
#define FIX_CASE(R) \
    case R: pass0<R>(b0, p.n, lb, sm, p.np, get); break;
        FIX_RADICES(FIX_CASE)
#undef FIX_CASE
    }
    __syncthreads();
    I2 *src = b0, *dst = b1;
    int Ns = p.r[0];
    for (int q = 1; q < p.np; ++q) {
        switch (p.r[q]) {
#define FIX_CASE(R) \
    case R: pass<R>(src, dst, p.n, lb, Ns, p.tw, sm, q == 1); break;
            FIX_RADICES(FIX_CASE)
#undef FIX_CASE
        }
        __syncthreads();
        Ns *= p.r[q];
        I2* t = src;
        src = dst;
        dst = t;
    }
    return src;
}

struct RowArgs {
    const double* re[kMaxFields];  // real fields (in: r2c, out: c2r)
    double2* sp[kMaxFields];       // half spectra
    Grid3 g;
    int lb;           // log2 of the lines (row pairs) per tile
    FastDiv dn, dh;   // by n2 and n2h
};

// R2C along axis 2: 2 L rows per block
static __global__ void __launch_bounds__(kThreads, 3) k_rows_r2c(RowArgs a) {
    extern __shared__ __align__(16) unsigned char fix_smem[];
    __shared__ LineSm sm;
    const int n = a.g.n2, h = a.g.n2h, L = 1 << a.lb, LP = L + 1;
    I2* b0 = reinterpret_cast<I2*>(fix_smem);
    I2* b1 = b0 + n * LP;
    const double* in = a.re[blockIdx.y];
    double2* out = a.sp[blockIdx.y];
    const long long rows = (long long)a.g.n0 * a.g.n1, row0 = (long long)blockIdx.x * 2 * L;
    const int nr = (int)min(2LL * L, rows - row0);
    double* raw = reinterpret_cast<double*>(b1);  // element (n, row r) at 2 (n LP + r / 2) + r % 2
    for (int e = threadIdx.x; e < 2 * L * n; e += kThreads) {
        const int r = a.dn.div(e), i = e - r * n;
        raw[2 * (i * LP + (r >> 1)) + (r & 1)] = r < nr ? in[(row0 + r) * n + i] : 0.0;
    }
    __syncthreads();
    const double2* raw2 = reinterpret_cast<const double2*>(b1);
    const I2* z = tile_fft(b0, b1, a.g.p2, a.lb, sm, [&](int i, int l) { return raw2[i * LP + l]; });
    // X_a = (Z + conj Z')/2, X_b = (Z - conj Z')/(2i), Z' = Z[n - k]
    for (int e = threadIdx.x; e < L * h; e += kThreads) {
        const int l = a.dh.div(e), k = e - l * h;
        const Scale c = sm.c[l];
        const int ds = sm.ds[l];
        const I2 Z = z[k * LP + l], Y = z[(k ? n - k : 0) * LP + l];
        const long long o = (row0 + 2 * l) * h + k;
        if (2 * l < nr)
            out[o] = make_double2(to_dbl(Z.x + Y.x, c, ds - 1), to_dbl(Z.y - Y.y, c, ds - 1));
        if (2 * l + 1 < nr)
            out[o + h] = make_double2(to_dbl(Z.y + Y.y, c, ds - 1), to_dbl(Y.x - Z.x, c, ds - 1));
    }
}

// C2R along axis 2, unnormalised; the imaginary parts of k2 = 0 and k2 = n2/2 are dropped
static __global__ void __launch_bounds__(kThreads, 3) k_rows_c2r(RowArgs a) {
    extern __shared__ __align__(16) unsigned char fix_smem[];
    __shared__ LineSm sm;
    const int n = a.g.n2, h = a.g.n2h, L = 1 << a.lb, LP = L + 1;
    I2* b0 = reinterpret_cast<I2*>(fix_smem);
    I2* b1 = b0 + n * LP;
    const double2* in = a.sp[blockIdx.y];
    double* out = const_cast<double*>(a.re[blockIdx.y]);
    const long long rows = (long long)a.g.n0 * a.g.n1, row0 = (long long)blockIdx.x * 2 * L;
    const int nr = (int)min(2LL * L, rows - row0);
    double2* raw = reinterpret_cast<double2*>(b1);
    // Z[k] = X_a + i X_b and Z[n-k] = conj X_a + i conj X_b, real and imaginary parts
    // exchanged (an inverse transform is the forward one with its parts exchanged)
    for (int e = threadIdx.x; e < L * h; e += kThreads) {
        const int l = a.dh.div(e), k = e - l * h;
        const long long o = (row0 + 2 * l) * h + k;
        double2 A = make_double2(0.0, 0.0), B = A;
        if (2 * l < nr) A = in[o];
        if (2 * l + 1 < nr) B = in[o + h];
        const bool edge = k == 0 || 2 * k == n;
        if (edge) A.y = B.y = 0.0;
        raw[k * LP + l] = make_double2(A.y + B.x, A.x - B.y);
        if (!edge) raw[(n - k) * LP + l] = make_double2(B.x - A.y, A.x + B.y);
    }
    __syncthreads();
    const I2* z = tile_fft(b0, b1, a.g.p2, a.lb, sm, [&](int i, int l) { return raw[i * LP + l]; });
    for (int e = threadIdx.x; e < 2 * L * n; e += kThreads) {
        const int r = a.dn.div(e), i = e - r * n, l = r >> 1;
        if (r >= nr) break;
        const Scale c = sm.c[l];
        const int ds = sm.ds[l];
        const I2 Z = z[i * LP + l];
        out[(row0 + r) * n + i] = to_dbl((r & 1) ? Z.x : Z.y, c, ds);
    }
}

struct ColArgs {
    double2* sp[kMaxFields];
    Grid3 g;
    int lb, ktiles;  // log2 of the lines per tile, k2 tiles per line set
    int inverse;
};

__device__ __forceinline__ double2 swapped(double2 v) { return make_double2(v.y, v.x); }

// columns along AXIS (1 or 0), forward or inverse, in place
template <int AXIS>
__global__ void __launch_bounds__(kThreads, 3) k_cols(ColArgs a) {
    extern __shared__ __align__(16) unsigned char fix_smem[];
    __shared__ LineSm sm;
    const Plan& p = AXIS == 1 ? a.g.p1 : a.g.p0;
    const int n = p.n, L = 1 << a.lb, LP = L + 1;
    I2* b0 = reinterpret_cast<I2*>(fix_smem);
    I2* b1 = b0 + n * LP;
    const int outer = blockIdx.x / a.ktiles, k2 = (blockIdx.x % a.ktiles) * L;
    const int nl = min(L, a.g.n2h - k2);
    const long long stride = AXIS == 1 ? a.g.n2h : (long long)a.g.n1 * a.g.n2h;
    double2* base = a.sp[blockIdx.y] + (AXIS == 1 ? (long long)outer * a.g.n1 : (long long)outer) * a.g.n2h + k2;
    const bool inv = a.inverse != 0;
    const I2* z = tile_fft(b0, b1, p, a.lb, sm, [&](int i, int l) {
        if (l >= nl) return make_double2(0.0, 0.0);
        const double2 v = base[i * stride + l];
        return inv ? swapped(v) : v;
    });
    for (int e = threadIdx.x; e < n * L; e += kThreads) {
        const int l = e & (L - 1), i = e >> a.lb;
        if (l >= nl) continue;
        const Scale c = sm.c[l];
        const int ds = sm.ds[l];
        const I2 Z = z[i * LP + l];
        const double2 v = make_double2(to_dbl(Z.x, c, ds), to_dbl(Z.y, c, ds));
        base[i * stride + l] = inv ? swapped(v) : v;
    }
}

// Lines per tile of one axis: fewer on a small grid, so that its tiles fill the SMs
inline int tile_lb(const Plan& p, long long lines, int sms) {
    int L = lines_of(p, 8);
    while (L > 2 && lines < (long long)L * 2 * sms) L >>= 1;
    int lb = 0;
    while ((1 << lb) < L) ++lb;
    return lb;
}

// Dynamic shared memory above 48 KB needs an opt-in per kernel: always the same size, so
// that calls from several threads agree (256-point tiles of eight lines and a table
// take 82 KB).
constexpr int kSmemMax = 96 * 1024;
template <class K>
inline void smem_optin(K kernel, size_t bytes) {
    OFDFT_REQUIRE(bytes <= kSmemMax, "integer-pipe transform: tile of %zu bytes", bytes);
    if (bytes > 40 * 1024)  // the kernels hold some static shared memory beside it
        OFDFT_CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax));
}

inline RowArgs row_args(const Grid3& g, int sms) {
    RowArgs a{};
    a.g = g;
    a.lb = tile_lb(g.p2, ((long long)g.n0 * g.n1 + 1) / 2, sms);
    a.dn = fast_div(g.n2);
    a.dh = fast_div(g.n2h);
    return a;
}
inline unsigned row_blocks(const RowArgs& a) {
    const long long pairs = ((long long)a.g.n0 * a.g.n1 + 1) / 2;
    return (unsigned)((pairs + (1 << a.lb) - 1) >> a.lb);
}
inline ColArgs col_args(const Grid3& g, int axis, int sms) {
    ColArgs a{};
    a.g = g;
    a.lb = tile_lb(axis == 1 ? g.p1 : g.p0, (long long)(axis == 1 ? g.n0 : g.n1) * g.n2h, sms);
    a.ktiles = (g.n2h + (1 << a.lb) - 1) >> a.lb;
    return a;
}
inline unsigned col_blocks(const ColArgs& a, int axis) { return (unsigned)(axis == 1 ? a.g.n0 : a.g.n1) * a.ktiles; }

// nf fields from rows of real values to half spectra, axis 2 only
inline void rows_r2c(const Grid3& g, int sms, const double* const* in, double2* const* out, int nf, cudaStream_t st) {
    RowArgs a = row_args(g, sms);
    for (int f = 0; f < nf; ++f) a.re[f] = in[f], a.sp[f] = out[f];
    const size_t smem = tile_smem(g.p2, 1 << a.lb);
    smem_optin(k_rows_r2c, smem);
    k_rows_r2c<<<dim3(row_blocks(a), nf), kThreads, smem, st>>>(a);
    OFDFT_LAUNCH_CHECK();
}
inline void rows_c2r(const Grid3& g, int sms, double2* const* in, double* const* out, int nf, cudaStream_t st) {
    RowArgs a = row_args(g, sms);
    for (int f = 0; f < nf; ++f) a.re[f] = out[f], a.sp[f] = in[f];
    const size_t smem = tile_smem(g.p2, 1 << a.lb);
    smem_optin(k_rows_c2r, smem);
    k_rows_c2r<<<dim3(row_blocks(a), nf), kThreads, smem, st>>>(a);
    OFDFT_LAUNCH_CHECK();
}
template <int AXIS>
inline void cols(const Grid3& g, int sms, double2* const* sp, int nf, bool inverse, cudaStream_t st) {
    ColArgs a = col_args(g, AXIS, sms);
    for (int f = 0; f < nf; ++f) a.sp[f] = sp[f];
    a.inverse = inverse;
    const size_t smem = tile_smem(AXIS == 1 ? g.p1 : g.p0, 1 << a.lb);
    smem_optin(k_cols<AXIS>, smem);
    k_cols<AXIS><<<dim3(col_blocks(a, AXIS), nf), kThreads, smem, st>>>(a);
    OFDFT_LAUNCH_CHECK();
}

}  // namespace fix
}  // namespace ofdft
