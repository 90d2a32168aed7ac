// Three-dimensional float64 real transforms on the integer pipe (fix_fft.cuh): tiles
// of lines in shared memory, one block per tile, three axis passes per transform.
//   rows     axis 2: two adjacent rows as one complex line, split into (or joined
//            from) their half spectra
//   columns  axes 1 and 0, in place: a tile is L consecutive lines, numbered through
//            all (outer, k2), so no tile is padded but the last
// A launch covers several fields (blockIdx.y), each a half-complex array in cuFFT's
// R2C layout.  The first pass reads its elements straight into the registers of its
// butterflies, exchanges go through one shared buffer of the tile (read, barrier, write),
// and the last pass of a column hands its outputs to the caller from registers.
//
// What bounds it: neither a pipe (k_cols at 128^3: ALU 39, FP64 37, FMA 15% busy, issue slots
// 37%) nor memory (11%), but latency: straight-line butterflies of up to 16 elements on a dozen
// warps per SM, and instruction fetches.  Hence the small blocks with every thread busy and 128
// registers per thread.  128^3, three fields: one axis pass 52 us, the axis-0 pair with its factor
// 205 us, rows 73 and 78 us (a cuFFT float64 transform of one field takes 240 us; tiles padded
// along k2, two buffers and 168 registers per thread took 79, 291, 85 and 88 us).
#pragma once
#include "common.cuh"
#include "fix_fft.cuh"

namespace ofdft {
namespace fix {

constexpr int kThreads = 128;  // most threads of a tile
constexpr int kMaxLines = 16;
constexpr int kMaxFields = 8;
constexpr int kBlocks = 4;  // blocks per SM (128 registers per thread; 3 and 5 ran 5% slower)

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
    int emax[kMaxLines];
    unsigned most[kMaxLines];  // largest 1-norm of a first-pass subset
    unsigned sum[kMaxLines];   // 1-norm of the line
    int k[kMaxLines];          // fix_shift of the first pass
    int ds[kMaxLines];         // shift after it
};

// ---- passes.  A tile holds L = 2^lb lines; element n of line l sits at n (L + 1) + l.

// an output of a line with first-pass shift k and later shift ds (adj: a further power of two)
__device__ __forceinline__ double2 from_fix(I2 v, const LineSm& sm, int l, int adj = 0) {
    const int k = sm.ds[l] + adj - sm.k[l];
    const bool nan = sm.emax[l] == kNonFinite;
    return make_double2(to_dbl(v.x, k, nan), to_dbl(v.y, k, nan));
}

// The scales of the tile's lines from the elements that its threads hold (thread (j, l):
// elements v of line l), and v in fixed point; np, r1: passes of the transform and radix of
// the second one's (for the shift).  Two barriers; sm is reset by the caller.
template <int R>
__device__ __forceinline__ void agree(const double2 (&v)[R], I2 (&u)[R], bool on, int j, int l, LineSm& sm, int np) {
    int em = 0;
#pragma unroll
    for (int q = 0; q < R; ++q) em = max(em, max(expo(v[q].x), expo(v[q].y)));
    if (on) atomicMax(&sm.emax[l], em);
    __syncthreads();
    em = sm.emax[l];
    unsigned s = 0;
#pragma unroll
    for (int q = 0; q < R; ++q) s += bound(expo(v[q].x), em) + bound(expo(v[q].y), em);
    if (on) {
        atomicMax(&sm.most[l], s);
        atomicAdd(&sm.sum[l], s);
    }
    __syncthreads();
    const Scale c = scale_of(em, sm.most[l]);
    const int k = fix_shift(c);
    if (j == 0) {
        sm.k[l] = k;
        sm.ds[l] = later_shift(c, sm.sum[l], np);
    }
#pragma unroll
    for (int q = 0; q < R; ++q) u[q] = I2{to_fix(v[q].x, k), to_fix(v[q].y, k)};
}

__device__ __forceinline__ void reset(LineSm& sm) {
    if (threadIdx.x < kMaxLines) {
        sm.emax[threadIdx.x] = 0;
        sm.most[threadIdx.x] = 0;
        sm.sum[threadIdx.x] = 0;
    }
}

// First pass (radix R): elements from get(n, l) (float64 pairs), outputs into the buffer
template <int R, class Get>
__device__ __forceinline__ void pass0(I2* buf, int n, int lb, LineSm& sm, int np, Get get) {
    const int m = n / R, L = 1 << lb, l = threadIdx.x & (L - 1), j = threadIdx.x >> lb;
    const bool on = j < m;
    // a thread without a butterfly repeats butterfly 0 and stores nothing: with the elements
    // defined on some paths only, they are live around a caller's loop over tiles, and spilled
    const int i = on ? j : 0;
    double2 v[R];
    I2 u[R];
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = get(i + q * m, l);
    agree<R>(v, u, on, j, l, sm, np);
    Dft<R>::run(u);
    if (on) {
#pragma unroll
        for (int q = 0; q < R; ++q) buf[(j * R + q) * (L + 1) + l] = u[q];
    }
}

// inputs of butterfly j of a later pass (sub-transform length Ns), shifted and twiddled
template <int R>
__device__ __forceinline__ void gather(I2 (&u)[R], const I2* buf, int n, int lb, int Ns, int j, int l, int d,
                                       const Tw* __restrict__ tw) {
    const int m = n / R, LP = (1 << lb) + 1, step = (j % Ns) * (n / (Ns * R));
#pragma unroll
    for (int q = 0; q < R; ++q) {
        u[q] = buf[(j + q * m) * LP + l];
        if (q > 0) {
            const int4 w = __ldg(reinterpret_cast<const int4*>(tw) + q * step);
            u[q] = cmul(u[q], Tw{w.x, w.y, w.z, w.w});
        }
        u[q] = I2{shr(u[q].x, d), shr(u[q].y, d)};
    }
}

// Later pass from one buffer to the other
template <int R>
__device__ __forceinline__ void pass(const I2* src, I2* dst, int n, int lb, int Ns, const Tw* __restrict__ tw,
                                     const LineSm& sm, int q, int np, int r1) {
    const int L = 1 << lb, items = (n / R) << lb;
    for (int it = threadIdx.x; it < items; it += blockDim.x) {
        const int l = it & (L - 1), j = it >> lb;
        I2 u[R];
        gather<R>(u, src, n, lb, Ns, j, l, pass_shift(sm.ds[l], q, np, r1), tw);
        Dft<R>::run(u);
        const int base = (j / Ns) * Ns * R + j % Ns;
#pragma unroll
        for (int k = 0; k < R; ++k) dst[(base + k * Ns) * (L + 1) + l] = u[k];
    }
}

// Last pass, outputs to put(k, l, value)
template <int R, class Put>
__device__ __forceinline__ void pass_out(const I2* buf, int n, int lb, const Tw* __restrict__ tw, const LineSm& sm, int q,
                                         int np, int r1, Put put) {
    const int L = 1 << lb, m = n / R, items = m << lb;
    for (int it = threadIdx.x; it < items; it += blockDim.x) {
        const int l = it & (L - 1), j = it >> lb;
        I2 u[R];
        gather<R>(u, buf, n, lb, m, j, l, pass_shift(sm.ds[l], q, np, r1), tw);
        Dft<R>::run(u);
#pragma unroll
        for (int k = 0; k < R; ++k) put(j + k * m, l, u[k]);
    }
}

#define FIX_RADICES(CASE) \
    CASE(2) CASE(3) CASE(4) CASE(5) CASE(6) CASE(7) CASE(8) CASE(9) CASE(10) CASE(12) CASE(14) CASE(15) CASE(16)

// Passes 1 .. to - 1 of the plan (or of the plan with its radices reversed), from buffer to
// buffer; returns the one that holds the result
__device__ __forceinline__ I2* middle(I2* src, I2* dst, const Plan& p, int lb, const LineSm& sm, int to, bool reversed) {
    int Ns = reversed ? p.r[p.np - 1] : p.r[0];
    const int r1 = reversed ? p.r[p.np > 1 ? p.np - 2 : 0] : p.r[1];
    for (int q = 1; q < to; ++q) {
        const int R = reversed ? p.r[p.np - 1 - q] : p.r[q];
        switch (R) {
#define FIX_CASE(R_) \
    case R_: pass<R_>(src, dst, p.n, lb, Ns, p.tw, sm, q, p.np, r1); break;
            FIX_RADICES(FIX_CASE)
#undef FIX_CASE
        }
        __syncthreads();
        Ns *= R;
        I2* t = src;
        src = dst;
        dst = t;
    }
    return src;
}

// Transforms the tile's lines; returns the buffer with the result (visible to all).  Entry: no
// thread still uses sm; get may read b1 (the first pass writes b0 after every get).
template <class Get>
__device__ __forceinline__ const I2* tile_fft(I2* b0, I2* b1, const Plan& p, int lb, LineSm& sm, Get get) {
    reset(sm);
    __syncthreads();
    switch (p.r[0]) {
#define FIX_CASE(R) \
    case R: pass0<R>(b0, p.n, lb, sm, p.np, get); break;
        FIX_RADICES(FIX_CASE)
#undef FIX_CASE
    }
    __syncthreads();
    return middle(b0, b1, p, lb, sm, p.np, false);
}

// The same, every output to put(k, l, value) once; b1 is used by plans of three passes only
template <class Get, class Put>
__device__ __forceinline__ void tile_fft_out(I2* b0, I2* b1, const Plan& p, int lb, LineSm& sm, Get get, Put put) {
    reset(sm);
    __syncthreads();
    switch (p.r[0]) {
#define FIX_CASE(R) \
    case R: pass0<R>(b0, p.n, lb, sm, p.np, get); break;
        FIX_RADICES(FIX_CASE)
#undef FIX_CASE
    }
    __syncthreads();
    if (p.np == 1) {
        for (int e = threadIdx.x; e < p.n << lb; e += blockDim.x) {
            const int l = e & ((1 << lb) - 1), k = e >> lb;
            put(k, l, b0[k * ((1 << lb) + 1) + l]);
        }
        return;
    }
    const I2* z = middle(b0, b1, p, lb, sm, p.np - 1, false);
    switch (p.r[p.np - 1]) {
#define FIX_CASE(R) \
    case R: pass_out<R>(z, p.n, lb, p.tw, sm, p.np - 1, p.np, p.r[1], put); break;
        FIX_RADICES(FIX_CASE)
#undef FIX_CASE
    }
}

// ---- launch shapes
struct Shape {
    int lb, threads;
};
// Lines per tile and threads: one first-pass butterfly per thread (of the last radix too
// when `both`: a transform followed by its reversed inverse); among 16, 8, 4, 2 and 1 lines
// the most evenly used threads, and fewer lines on a grid too small to give every SM a few
// tiles.
inline Shape shape_of(const Plan& p, long long lines, int sms, bool both = false) {
    Shape best{0, 32};
    double score = -1.0;
    for (int lb = 4; lb >= 0; --lb) {
        const int L = 1 << lb;
        int need = L * (p.n / p.r[0]);
        if (both) need = std::max(need, L * (p.n / p.r[p.np - 1]));
        const int threads = (need + 31) / 32 * 32;
        if (threads > kThreads) continue;
        double use = 0.0;
        for (int q = 0; q < p.np; ++q) {
            const int items = L * (p.n / p.r[q]);
            use += (double)items / (((items + threads - 1) / threads) * threads) / p.np;
        }
        if (L < 8) use *= 0.5 * (0.5 + 0.125 * L);  // elements of 16 bytes: below a 128-byte segment
        if (lines < (long long)L * 2 * sms) use *= (double)lines / ((double)L * 2 * sms);
        if (use > score + 0.02) {
            score = use;
            best = Shape{lb, threads};
        }
    }
    return best;
}
// shared memory of a tile with `bufs` buffers (three-pass plans always take two)
inline size_t tile_smem(const Plan& p, int lb, int bufs) {
    return (size_t)(p.np == 3 ? 2 : bufs) * p.n * ((1 << lb) + 1) * sizeof(I2);
}

// Dynamic shared memory above 48 KB needs an opt-in per kernel: always the same size, so
// that calls from several threads agree (256 elements of 16 lines take 70 KB).
constexpr int kSmemMax = 160 * 1024;
template <class K>
inline void smem_optin(K kernel, size_t bytes) {
    OFDFT_REQUIRE(bytes <= kSmemMax, "integer-pipe transform: tile of %zu bytes", bytes);
    if (bytes > 40 * 1024)  // the kernels hold some static shared memory beside it
        OFDFT_CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax));
}

// ---- axis 2
struct RowArgs {
    const double* re[kMaxFields];  // real fields (in: r2c, out: c2r)
    double2* sp[kMaxFields];       // half spectra
    Grid3 g;
    int lb;           // log2 of the lines (row pairs) per tile
    FastDiv dn, dh;   // by n2 and n2h
};

// R2C along axis 2: 2 L rows per block
static __global__ void __launch_bounds__(kThreads, kBlocks) k_rows_r2c(RowArgs a) {
    extern __shared__ __align__(16) unsigned char fix_smem[];
    __shared__ LineSm sm;
    const int n = a.g.n2, h = a.g.n2h, L = 1 << a.lb, LP = L + 1, T = blockDim.x;
    I2* b0 = reinterpret_cast<I2*>(fix_smem);
    I2* b1 = b0 + n * LP;
    const double* in = a.re[blockIdx.y];
    double2* out = a.sp[blockIdx.y];
    const long long rows = (long long)a.g.n0 * a.g.n1, row0 = (long long)blockIdx.x * 2 * L;
    const int nr = (int)min(2LL * L, rows - row0);
    double* raw = reinterpret_cast<double*>(b1);  // element (n, row r) at 2 (n LP + r / 2) + r % 2
    for (int e = threadIdx.x; e < 2 * L * n; e += T) {
        const int r = a.dn.div(e), i = e - r * n;
        raw[2 * (i * LP + (r >> 1)) + (r & 1)] = r < nr ? in[(row0 + r) * n + i] : 0.0;
    }
    __syncthreads();
    const double2* raw2 = reinterpret_cast<const double2*>(b1);
    const I2* buf = tile_fft(b0, b1, a.g.p2, a.lb, sm, [&](int i, int l) { return raw2[i * LP + l]; });
    // X_a = (Z + conj Z')/2, X_b = (Z - conj Z')/(2i), Z' = Z[n - k]
    for (int e = threadIdx.x; e < L * h; e += T) {
        const int l = a.dh.div(e), k = e - l * h;
        const I2 Z = buf[k * LP + l], Y = buf[(k ? n - k : 0) * LP + l];
        const long long o = (row0 + 2 * l) * h + k;
        if (2 * l < nr) out[o] = from_fix(I2{Z.x + Y.x, Z.y - Y.y}, sm, l, -1);
        if (2 * l + 1 < nr) out[o + h] = from_fix(I2{Z.y + Y.y, Y.x - Z.x}, sm, l, -1);
    }
}

// Two half-spectrum rows joined into one complex line, real and imaginary parts exchanged (an
// inverse transform is the forward one with its parts exchanged): Z[k] = X_a + i X_b,
// Z[n-k] = conj X_a + i conj X_b; the imaginary parts of k2 = 0 and k2 = n2/2 are dropped
__device__ __forceinline__ void join_rows(double2* raw, double2 A, double2 B, int k, int l, int n, int LP) {
    const bool edge = k == 0 || 2 * k == n;
    if (edge) A.y = B.y = 0.0;
    raw[k * LP + l] = make_double2(A.y + B.x, A.x - B.y);
    if (!edge) raw[(n - k) * LP + l] = make_double2(B.x - A.y, A.x + B.y);
}

// C2R along axis 2, unnormalised
static __global__ void __launch_bounds__(kThreads, kBlocks) k_rows_c2r(RowArgs a) {
    extern __shared__ __align__(16) unsigned char fix_smem[];
    __shared__ LineSm sm;
    const int n = a.g.n2, h = a.g.n2h, L = 1 << a.lb, LP = L + 1, T = blockDim.x;
    I2* b0 = reinterpret_cast<I2*>(fix_smem);
    I2* b1 = b0 + n * LP;
    const double2* in = a.sp[blockIdx.y];
    double* out = const_cast<double*>(a.re[blockIdx.y]);
    const long long rows = (long long)a.g.n0 * a.g.n1, row0 = (long long)blockIdx.x * 2 * L;
    const int nr = (int)min(2LL * L, rows - row0);
    double2* raw = reinterpret_cast<double2*>(b1);
    for (int e = threadIdx.x; e < L * h; e += T) {
        const int l = a.dh.div(e), k = e - l * h;
        const long long o = (row0 + 2 * l) * h + k;
        double2 A = make_double2(0.0, 0.0), B = A;
        if (2 * l < nr) A = in[o];
        if (2 * l + 1 < nr) B = in[o + h];
        join_rows(raw, A, B, k, l, n, LP);
    }
    __syncthreads();
    const I2* buf = tile_fft(b0, b1, a.g.p2, a.lb, sm, [&](int i, int l) { return raw[i * LP + l]; });
    for (int e = threadIdx.x; e < 2 * L * n; e += T) {
        const int r = a.dn.div(e), i = e - r * n, l = r >> 1;
        if (r >= nr) break;
        const I2 Z = buf[i * LP + l];
        out[(row0 + r) * n + i] = to_dbl((r & 1) ? Z.x : Z.y, sm.ds[l] - sm.k[l], sm.emax[l] == kNonFinite);
    }
}

// ---- axes 1 and 0
struct ColArgs {
    double2* sp[kMaxFields];
    Grid3 g;
    int lb;  // log2 of the lines per tile
    int inverse;
};

__device__ __forceinline__ double2 swapped(double2 v) { return make_double2(v.y, v.x); }

// offset of line `line` (numbered through (outer, k2)) of an axis
template <int AXIS>
__device__ __forceinline__ long long col_base(const Grid3& g, int line) {
    if (AXIS == 0) return line;
    const int i0 = line / g.n2h;
    return (long long)i0 * (g.n1 - 1) * g.n2h + line;
}
template <int AXIS>
__host__ __device__ __forceinline__ int col_lines(const Grid3& g) {
    return (AXIS == 1 ? g.n0 : g.n1) * g.n2h;
}
template <int AXIS>
__device__ __forceinline__ long long col_stride(const Grid3& g) {
    return AXIS == 1 ? g.n2h : (long long)g.n1 * g.n2h;
}

// columns along AXIS, forward or inverse, in place
template <int AXIS>
__global__ void __launch_bounds__(kThreads, kBlocks) k_cols(ColArgs a) {
    extern __shared__ __align__(16) unsigned char fix_smem[];
    __shared__ LineSm sm;
    const Plan& p = AXIS == 1 ? a.g.p1 : a.g.p0;
    I2* b0 = reinterpret_cast<I2*>(fix_smem);
    // a thread's line: the same in every pass (the threads are a multiple of the lines)
    const int line = (blockIdx.x << a.lb) + (threadIdx.x & ((1 << a.lb) - 1));
    const bool in = line < col_lines<AXIS>(a.g);
    const long long stride = col_stride<AXIS>(a.g);
    double2* base = a.sp[blockIdx.y] + (in ? col_base<AXIS>(a.g, line) : 0);
    const bool inv = a.inverse != 0;
    tile_fft_out(
        b0, b0 + p.n * ((1 << a.lb) + 1), p, a.lb, sm,
        [&](int i, int) {
            if (!in) return make_double2(0.0, 0.0);
            const double2 v = base[i * stride];
            return inv ? swapped(v) : v;
        },
        [&](int i, int l, I2 z) {
            if (!in) return;
            const double2 v = from_fix(z, sm, l);
            base[i * stride] = inv ? swapped(v) : v;
        });
}

// ---- launches
inline RowArgs row_args(const Grid3& g, const Shape& s) {
    RowArgs a{};
    a.g = g;
    a.lb = s.lb;
    a.dn = fast_div(g.n2);
    a.dh = fast_div(g.n2h);
    return a;
}
inline Shape row_shape(const Grid3& g, int sms) { return shape_of(g.p2, ((long long)g.n0 * g.n1 + 1) / 2, sms); }
inline unsigned row_blocks(const Grid3& g, int lb) {
    const long long pairs = ((long long)g.n0 * g.n1 + 1) / 2;
    return (unsigned)((pairs + (1 << lb) - 1) >> lb);
}
inline unsigned col_blocks(int lines, int lb) { return (unsigned)(((long long)lines + (1 << lb) - 1) >> lb); }

// nf fields from rows of real values to half spectra, axis 2 only
inline void rows_r2c(const Grid3& g, int sms, const double* const* in, double2* const* out, int nf, cudaStream_t st) {
    const Shape s = row_shape(g, sms);
    RowArgs a = row_args(g, s);
    for (int f = 0; f < nf; ++f) a.re[f] = in[f], a.sp[f] = out[f];
    const size_t smem = tile_smem(g.p2, s.lb, 2);
    smem_optin(k_rows_r2c, smem);
    k_rows_r2c<<<dim3(row_blocks(g, s.lb), nf), s.threads, smem, st>>>(a);
    OFDFT_LAUNCH_CHECK();
}
inline void rows_c2r(const Grid3& g, int sms, double2* const* in, double* const* out, int nf, cudaStream_t st) {
    const Shape s = row_shape(g, sms);
    RowArgs a = row_args(g, s);
    for (int f = 0; f < nf; ++f) a.re[f] = out[f], a.sp[f] = in[f];
    const size_t smem = tile_smem(g.p2, s.lb, 2);
    smem_optin(k_rows_c2r, smem);
    k_rows_c2r<<<dim3(row_blocks(g, s.lb), nf), s.threads, smem, st>>>(a);
    OFDFT_LAUNCH_CHECK();
}
template <int AXIS>
inline void cols(const Grid3& g, int sms, double2* const* sp, int nf, bool inverse, cudaStream_t st) {
    const Plan& p = AXIS == 1 ? g.p1 : g.p0;
    const Shape s = shape_of(p, col_lines<AXIS>(g), sms);
    ColArgs a{};
    a.g = g;
    a.lb = s.lb;
    a.inverse = inverse;
    for (int f = 0; f < nf; ++f) a.sp[f] = sp[f];
    const size_t smem = tile_smem(p, s.lb, 1);
    smem_optin(k_cols<AXIS>, smem);
    k_cols<AXIS><<<dim3(col_blocks(col_lines<AXIS>(g), s.lb), nf), s.threads, smem, st>>>(a);
    OFDFT_LAUNCH_CHECK();
}

}  // namespace fix
}  // namespace ofdft
