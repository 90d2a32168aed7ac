// Float64 line FFTs on the integer pipe.
//
// GB300 issues two float64 operations per SM and clock, 1/64 of its float32 rate
// and 1/32 of its 32-bit integer rate, and a float64 FFT is mostly additions.
// These transforms therefore run in block fixed point: a line is converted to
// 64-bit integers with one power-of-two scale, transformed with integer
// additions and 64-bit fixed-point products, and converted back.
//
// Precision.  With R the first pass's radix, the scale maps the largest 1-norm
// sum |re| + |im| of the subsets that the first pass transforms (every (n/R)-th
// element) to at most 2^61, and the later passes' sums, up to the line's whole 1-norm,
// to at most 2^61 as well.  The norms are bounds from the elements' exponents; elements 22
// binades or more below the line's largest count as nothing, which leaves out less than
// 2^-12 of the norm and is covered by the room up to 2^62 that the products have.  Every
// intermediate of an FFT is a sum of the inputs with weights of modulus one, so none
// exceeds these bounds: nothing overflows, and no bits are given up that the line's
// own values do not need.  For flat lines of up to 512 elements the unit is 2^-56 of
// the mean element in the first pass and 2^-52 of the mean element, 2^-56 of the mean
// output, after it; for a line with one dominant element it is 2^-61 of that.  That
// is below the rounding of a float64 FFT, whose every addition rounds to 2^-53 of the
// partial sum.  Twiddles carry 61 bits; elements are rounded to float64 once, on return.
//
// A line with an infinity or a NaN returns NaN in every element; subnormal
// inputs count as zero.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace ofdft {
namespace fix {

#define FIX_HD __host__ __device__ __forceinline__

struct __align__(16) I2 {
    long long x, y;
};

FIX_HD I2 operator+(I2 a, I2 b) { return I2{a.x + b.x, a.y + b.y}; }
FIX_HD I2 operator-(I2 a, I2 b) { return I2{a.x - b.x, a.y - b.y}; }
FIX_HD I2 mul_mi(I2 a) { return I2{a.y, -a.x}; }  // times -i

// 31-bit limbs: v = h 2^31 + l, 0 <= l < 2^31 (|v| < 2^62)
FIX_HD int hi31(long long v) { return (int)(v >> 31); }
FIX_HD int lo31(long long v) { return (int)(v & 0x7fffffffLL); }

// x c 2^-61: the product of the low limbs (less than two units) is dropped
FIX_HD long long mulc(long long x, long long c) {
    const int xh = hi31(x), xl = lo31(x), ch = hi31(c), cl = lo31(c);
    return 2 * ((long long)xh * ch) + (((long long)xh * cl + (long long)xl * ch) >> 30);
}
FIX_HD I2 mulr(I2 a, long long c) { return I2{mulc(a.x, c), mulc(a.y, c)}; }
FIX_HD I2 half(I2 a) { return I2{a.x >> 1, a.y >> 1}; }
FIX_HD I2 quarter(I2 a) { return I2{a.x >> 2, a.y >> 2}; }

// a twiddle at scale 2^61 in 31-bit limbs: real part high, low, imaginary part high, low
struct __align__(16) Tw {
    int ch, cl, dh, dl;
};
FIX_HD Tw tw_of(long long re, long long im) { return Tw{hi31(re), lo31(re), hi31(im), lo31(im)}; }

FIX_HD I2 cmul(I2 x, Tw w) {
    const int ah = hi31(x.x), al = lo31(x.x), bh = hi31(x.y), bl = lo31(x.y);
    const int ch = w.ch, cl = w.cl, dh = w.dh, dl = w.dl;
    const long long ac = (long long)ah * cl + (long long)al * ch, bd = (long long)bh * dl + (long long)bl * dh;
    const long long x2 = (long long)ah * dl + (long long)al * dh + (long long)bh * cl + (long long)bl * ch;
    const long long re = (long long)ah * ch - (long long)bh * dh;
    const long long im = (long long)ah * dh + (long long)bh * ch;
    return I2{2 * re + ((ac - bd) >> 30), 2 * im + (x2 >> 30)};
}

// cos and sin of 2 pi k / n at scale 2^61
constexpr long long kOne = 1LL << 61;
constexpr long long kS3 = 1996918623117814388LL;                                        // sin(2 pi/3)
constexpr long long kR5 = 1289005428511123393LL;                                        // sqrt(5)/4
constexpr long long kS51 = 2192987019466309470LL, kS52 = 1355340514917506542LL;         // sin(2 pi k/5)
constexpr long long kH = 1630477228166597777LL;                                         // sqrt(1/2)
constexpr long long kC71 = 1437669600931991917LL, kC72 = -513098339966869658LL, kC73 = -2077492765571969234LL;
constexpr long long kS71 = 1802780658232085260LL, kS72 = 2248030710791760100LL, kS73 = 1000467786655719552LL;
constexpr long long kC91 = 1766378223912892722LL, kC92 = 400405436535988841LL, kC94 = -2166783660448881563LL;
constexpr long long kS91 = 1482167316204887212LL, kS92 = 2270812072702646106LL, kS94 = 788644756497758894LL;
constexpr long long kC161 = 2130321161396766249LL, kS161 = 882407917260943721LL;        // cos, sin(pi/8)

// ---- forward DFTs of R points in registers, natural order in and out
template <int R>
struct Dft;

template <>
struct Dft<2> {
    FIX_HD static void run(I2* u) {
        const I2 a = u[0];
        u[0] = a + u[1];
        u[1] = a - u[1];
    }
};
template <>
struct Dft<3> {
    FIX_HD static void run(I2* u) {
        const I2 s = u[1] + u[2], t = mul_mi(mulr(u[1] - u[2], kS3)), m = u[0] - half(s);
        u[0] = u[0] + s;
        u[1] = m + t;
        u[2] = m - t;
    }
};
template <>
struct Dft<4> {
    FIX_HD static void run(I2* u) {
        const I2 a = u[0] + u[2], b = u[0] - u[2], c = u[1] + u[3], d = mul_mi(u[1] - u[3]);
        u[0] = a + c;
        u[2] = a - c;
        u[1] = b + d;
        u[3] = b - d;
    }
};
// five points: the cosine sums through (c1 - c2)/2 = sqrt(5)/4, the sine sums with three products
template <>
struct Dft<5> {
    FIX_HD static void run(I2* u) {
        const I2 a1 = u[1] + u[4], b1 = u[1] - u[4], a2 = u[2] + u[3], b2 = u[2] - u[3];
        const I2 t = a1 + a2, r = u[0] - quarter(t), s = mulr(a1 - a2, kR5);
        const I2 p = mulr(b1 + b2, kS52);
        const I2 i1 = mul_mi(p + mulr(b1, kS51 - kS52)), i2 = mul_mi(p - mulr(b2, kS51 + kS52));
        const I2 r1 = r + s, r2 = r - s;
        u[0] = u[0] + t;
        u[1] = r1 + i1;
        u[4] = r1 - i1;
        u[2] = r2 + i2;
        u[3] = r2 - i2;
    }
};
// seven points after Winograd: eight real products per component
template <>
struct Dft<7> {
    FIX_HD static void run(I2* u) {
        const I2 t1 = u[1] + u[6], t2 = u[2] + u[5], t3 = u[3] + u[4];
        const I2 t5 = u[1] - u[6], t6 = u[2] - u[5], t7 = u[4] - u[3];
        const I2 t4 = t1 + t2 + t3;
        const I2 t8 = t1 - t3, t9 = t3 - t2, t11 = t7 - t5, t12 = t6 - t7;
        const I2 m1 = mulr(t8, (2 * kC71 - kC72 - kC73) / 3), m2 = mulr(t9, (kC71 - 2 * kC72 + kC73) / 3);
        const I2 m3 = mulr(t2 - t1, (kC71 + kC72 - 2 * kC73) / 3);
        const I2 m4 = mulr(t5 + t6 + t7, (kS71 + kS72 - kS73) / 3);
        const I2 m5 = mulr(t11, (2 * kS71 - kS72 + kS73) / 3), m6 = mulr(t12, (kS71 - 2 * kS72 - kS73) / 3);
        const I2 m7 = mulr(t5 - t6, (kS71 + kS72 + 2 * kS73) / 3);
        const I2 s5 = u[0] - mulr(t4, kOne / 6);
        u[0] = u[0] + t4;
        const I2 r1 = s5 + m1 + m2, r2 = s5 - m1 - m3, r3 = s5 - m2 + m3;
        const I2 i1 = mul_mi(m4 - m5 - m6), i2 = mul_mi(m4 + m5 + m7), i3 = mul_mi(m6 - m7 + m4);
        u[1] = r1 + i1;
        u[6] = r1 - i1;
        u[2] = r2 + i2;
        u[5] = r2 - i2;
        u[3] = r3 - i3;
        u[4] = r3 + i3;
    }
};
template <>
struct Dft<8> {
    FIX_HD static void run(I2* u) {
        I2 e[4] = {u[0], u[2], u[4], u[6]}, o[4] = {u[1], u[3], u[5], u[7]};
        Dft<4>::run(e);
        Dft<4>::run(o);
        // w8 (x + iy) = sqrt(1/2) ((x + y) + i (y - x)), w8^3 = -i w8
        const I2 w1 = I2{mulc(o[1].x + o[1].y, kH), mulc(o[1].y - o[1].x, kH)};
        const I2 w2 = mul_mi(o[2]);
        const I2 w3 = I2{mulc(o[3].y - o[3].x, kH), mulc(-(o[3].x + o[3].y), kH)};
        u[0] = e[0] + o[0];
        u[4] = e[0] - o[0];
        u[1] = e[1] + w1;
        u[5] = e[1] - w1;
        u[2] = e[2] + w2;
        u[6] = e[2] - w2;
        u[3] = e[3] + w3;
        u[7] = e[3] - w3;
    }
};
template <>
struct Dft<9> {
    FIX_HD static void run(I2* u) {
        I2 a[3][3];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
#pragma unroll
            for (int r = 0; r < 3; ++r) a[j][r] = u[j + 3 * r];
            Dft<3>::run(a[j]);
        }
        a[1][1] = cmul(a[1][1], tw_of(kC91, -kS91));
        a[1][2] = cmul(a[1][2], tw_of(kC92, -kS92));
        a[2][1] = cmul(a[2][1], tw_of(kC92, -kS92));
        a[2][2] = cmul(a[2][2], tw_of(kC94, -kS94));
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            I2 b[3] = {a[0][k], a[1][k], a[2][k]};
            Dft<3>::run(b);
#pragma unroll
            for (int q = 0; q < 3; ++q) u[k + 3 * q] = b[q];
        }
    }
};
template <>
struct Dft<16> {
    FIX_HD static void run(I2* u) {
        I2 a[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
#pragma unroll
            for (int r = 0; r < 4; ++r) a[j][r] = u[j + 4 * r];
            Dft<4>::run(a[j]);
        }
        const Tw w1 = tw_of(kC161, -kS161), w3 = tw_of(kS161, -kC161), w9 = tw_of(-kC161, kS161);
        auto w2 = [](I2 v) { return I2{mulc(v.x + v.y, kH), mulc(v.y - v.x, kH)}; };
        auto w6 = [](I2 v) { return I2{mulc(v.y - v.x, kH), mulc(-(v.x + v.y), kH)}; };
        a[1][1] = cmul(a[1][1], w1);
        a[1][2] = w2(a[1][2]);
        a[1][3] = cmul(a[1][3], w3);
        a[2][1] = w2(a[2][1]);
        a[2][2] = mul_mi(a[2][2]);
        a[2][3] = w6(a[2][3]);
        a[3][1] = cmul(a[3][1], w3);
        a[3][2] = w6(a[3][2]);
        a[3][3] = cmul(a[3][3], w9);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            I2 b[4] = {a[0][k], a[1][k], a[2][k], a[3][k]};
            Dft<4>::run(b);
#pragma unroll
            for (int q = 0; q < 4; ++q) u[k + 4 * q] = b[q];
        }
    }
};
// R = A B with coprime A, B (Good-Thomas): no twiddles.  Element (a, b) sits at
// (a B + b A) mod R; output (p, q) at the index congruent to p mod A and q mod B.
template <int A, int B>
struct DftPfa {
    static constexpr int R = A * B;
    FIX_HD static constexpr int out(int p, int q) {
        int k = 0;
        while (k % A != p || k % B != q) ++k;
        return k;
    }
    template <int P, int Q>
    FIX_HD static void put(I2* u, const I2 (&a)[B][A]) {
        constexpr int k = out(P, Q);
        u[k] = a[Q][P];
        if constexpr (Q + 1 < B) put<P, Q + 1>(u, a);
        else if constexpr (P + 1 < A) put<P + 1, 0>(u, a);
    }
    FIX_HD static void run(I2* u) {
        I2 a[B][A];
#pragma unroll
        for (int b = 0; b < B; ++b) {
#pragma unroll
            for (int i = 0; i < A; ++i) a[b][i] = u[(i * B + b * A) % R];
            Dft<A>::run(a[b]);
        }
#pragma unroll
        for (int p = 0; p < A; ++p) {
            I2 c[B];
#pragma unroll
            for (int b = 0; b < B; ++b) c[b] = a[b][p];
            Dft<B>::run(c);
#pragma unroll
            for (int b = 0; b < B; ++b) a[b][p] = c[b];
        }
        put<0, 0>(u, a);
    }
};
template <>
struct Dft<6> : DftPfa<2, 3> {};
template <>
struct Dft<10> : DftPfa<2, 5> {};
template <>
struct Dft<12> : DftPfa<4, 3> {};
template <>
struct Dft<14> : DftPfa<2, 7> {};
template <>
struct Dft<15> : DftPfa<3, 5> {};

// ---- float64 <-> fixed point
FIX_HD unsigned long long bits_of(double v) {
#ifdef __CUDA_ARCH__
    return (unsigned long long)__double_as_longlong(v);
#else
    unsigned long long b;
    __builtin_memcpy(&b, &v, 8);
    return b;
#endif
}
FIX_HD double of_bits(unsigned long long b) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)b);
#else
    double v;
    __builtin_memcpy(&v, &b, 8);
    return v;
#endif
}
FIX_HD int expo(double v) { return (int)((unsigned)(bits_of(v) >> 52) & 0x7ffu); }  // biased exponent
// a bound of |v| in units of 2^(emax - 20), from its biased exponent e
FIX_HD unsigned bound(int e, int emax) {
    const int d = emax - e;
    return 0x200000u >> (d < 31 ? d : 31);
}
// The scale of a line: emax, the largest biased exponent, and sh, the bit length of a
// bound of the 1-norm in units of 2^(emax - 20).  x becomes x 2^(81 - sh) 2^-emax.
constexpr int kNonFinite = 0x7ff;
struct Scale {
    int emax, sh;
};
FIX_HD int bit_length(unsigned v) {  // 1 for 0
#ifdef __CUDA_ARCH__
    return 32 - __clz((int)(v | 1u));
#else
    return 32 - __builtin_clz(v | 1u);
#endif
}
// from the largest first-pass subset's bound, and the shift that the whole line's bound asks
// for after that pass
FIX_HD Scale scale_of(int emax, unsigned most) { return Scale{emax, bit_length(most)}; }
FIX_HD int later_shift(Scale s, unsigned sum, int np) { return np > 1 ? bit_length(sum) - s.sh : 0; }
// The shift in front of pass q >= 1 when the whole line needs ds: what the pass can grow
// by (ceil log2 of its radix), or what is left
FIX_HD int pass_shift(int ds, int q, int np, int r1) {
    const int grow = r1 > 8 ? 4 : (r1 > 4 ? 3 : (r1 > 2 ? 2 : 1));
    const int first = np == 2 || ds < grow ? ds : grow;
    return q == 1 ? first : ds - first;
}
// v 2^-d, rounded
FIX_HD long long shr(long long v, int d) { return (v + ((1LL << d) >> 1)) >> d; }
// 64-bit roundings between integers and float64
FIX_HD long long rint64(double v) {
#ifdef __CUDA_ARCH__
    return __double2ll_rn(v);
#else
    return __builtin_llrint(v);
#endif
}
// v at the line's scale: k = fix_shift is added to the exponent field (|v| 2^k' is below
// 2^62); a zero, subnormal or wrapping element becomes a tiny value, which rounds to 0
FIX_HD int fix_shift(Scale s) { return 81 - s.sh - s.emax + 1023; }
FIX_HD long long to_fix(double v, int k) {
    const unsigned long long b = bits_of(v);
    const int hi = (int)(b >> 32), e = (hi >> 20) & 0x7ff;
    const unsigned t = e == 0 || e + k <= 0 ? 0u : (unsigned)(hi + (k << 20));
    return rint64(of_bits(((unsigned long long)t << 32) | (b & 0xffffffffULL)));
}
// v 2^(k - 1023 + ...) for an output of the line: k = shift after the first pass - fix_shift;
// 0 on underflow, infinite on overflow, NaN in a line that was not finite
FIX_HD double to_dbl(long long v, int k, bool nan) {
    const unsigned long long b = bits_of((double)v);
    const int hi = (int)(b >> 32), e = ((hi >> 20) & 0x7ff) + k;
    unsigned t = (unsigned)(hi + (k << 20)), lo = (unsigned)b;
    if (v == 0 || e <= 0) t = lo = 0u;
    if (v != 0 && e >= 0x7ff) {
        t = (hi & 0x80000000u) | 0x7ff00000u;
        lo = 0u;
    }
    if (nan) t = 0x7ff80000u;
    return of_bits(((unsigned long long)t << 32) | lo);
}

// ---- plans: radices of a length, largest first where twiddles are fewest
constexpr int kMaxPass = 3;
// The longest line: its two bounds per element are added up in 32 bits.
constexpr int kMaxLen = 512;
static_assert(2ULL * kMaxLen * 0x200000u < 1ULL << 32, "the 1-norm's bound wraps");
struct Plan {
    int n = 0, np = 0;
    int r[kMaxPass] = {0, 0, 0};
    const Tw* tw = nullptr;  // exp(-2 pi i k/n), k < n
};

// false when n has a prime factor above 7, or is too long
inline bool plan_radices(int n, Plan& p) {
    static const int radix[13] = {16, 15, 14, 12, 10, 9, 8, 7, 6, 5, 4, 3, 2};
    if (n < 2 || n > kMaxLen) return false;
    p.n = n;
    p.np = 0;
    for (int a : radix)
        if (n == a) {
            p.np = 1;
            p.r[0] = n;
            return true;
        }
    // two passes: the most even split
    int best = 0;
    for (int a : radix)
        for (int b : radix)
            if (a >= b && a * b == n && (!best || a < best)) best = a;
    if (best) {
        // the larger radix first: the units of the second pass then grow by the smaller one
        p.np = 2;
        p.r[0] = best;
        p.r[1] = n / best;
        return true;
    }
    for (int a : radix)
        for (int b : radix)
            for (int c : radix)
                if (a >= b && b >= c && a * b * c == n && (!best || a < best)) {
                    best = a;
                    p.np = 3;
                    p.r[0] = a;
                    p.r[1] = b;
                    p.r[2] = c;
                }
    return best != 0;
}

}  // namespace fix
}  // namespace ofdft
