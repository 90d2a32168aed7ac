"""The scale of the integer-pipe transforms, by the functions that the kernels call, on lines that
reach its bounds: every length that has a plan, and none above."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include "fix_fft.cuh"
#include <algorithm>
#include <cmath>
#include <utility>
#include <vector>
using namespace ofdft::fix;
static void dft(int R, I2* u) {
    switch (R) {
#define C(r) case r: Dft<r>::run(u); break;
        C(2) C(3) C(4) C(5) C(6) C(7) C(8) C(9) C(10) C(12) C(14) C(15) C(16)
    }
}
// 0: no plan; *most: the largest |value| of any pass, before and after
extern "C" int line_fft(int n, const double* in, double* out, double* most) {
    Plan p;
    if (!plan_radices(n, p)) return 0;
    if (!in) return 1;
    std::vector<I2> a(n), b(n);
    std::vector<Tw> tw(n);
    for (int k = 0; k < n; ++k) {
        const long double t = -2.0L * 3.14159265358979323846264338327950288L * k / n;
        tw[k] = tw_of((long long)std::llroundl(std::cos(t) * (long double)kOne),
                      (long long)std::llroundl(std::sin(t) * (long double)kOne));
    }
    int em = 0;
    for (int i = 0; i < 2 * n; ++i) em = std::max(em, expo(in[i]));
    unsigned top = 0, sum = 0;
    for (int j = 0; j < n / p.r[0]; ++j) {
        unsigned s = 0;
        for (int q = 0; q < p.r[0]; ++q) {
            const double* v = in + 2 * (j + q * (n / p.r[0]));
            s += bound(expo(v[0]), em) + bound(expo(v[1]), em);
        }
        top = std::max(top, s);
        sum += s;
    }
    const Scale c = scale_of(em, top);
    const int ds = later_shift(c, sum, p.np), k = fix_shift(c);
    for (int i = 0; i < n; ++i) a[i] = I2{to_fix(in[2 * i], k), to_fix(in[2 * i + 1], k)};
    int Ns = 1;
    *most = 0.0;
    for (int q = 0; q < p.np; ++q) {
        const int R = p.r[q], m = n / R, step = n / (Ns * R);
        for (int j = 0; j < m; ++j) {
            I2 u[16];
            for (int r = 0; r < R; ++r) {
                u[r] = a[j + r * m];
                if (r && q) u[r] = cmul(u[r], tw[(j % Ns) * r * step]);
                if (q) {
                    const int d = pass_shift(ds, q, p.np, p.r[1]);
                    u[r] = I2{shr(u[r].x, d), shr(u[r].y, d)};
                }
            }
            dft(R, u);
            for (int r = 0; r < R; ++r) {
                b[(j / Ns) * Ns * R + j % Ns + r * Ns] = u[r];
                *most = std::max(*most, std::max(std::fabs((double)u[r].x), std::fabs((double)u[r].y)));
            }
        }
        std::swap(a, b);
        Ns *= R;
    }
    for (int i = 0; i < n; ++i) {
        out[2 * i] = to_dbl(a[i].x, ds - k, em == kNonFinite);
        out[2 * i + 1] = to_dbl(a[i].y, ds - k, em == kNonFinite);
    }
    return 1;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("scale")
    src, so = d / "line.cpp", d / "line.so"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I/usr/local/cuda/include",
                    "-I" + os.path.join(REPO, "dftpy_gb300", "csrc"), "-o", str(so), str(src)], check=True)
    lib = C.CDLL(str(so))
    lib.line_fft.argtypes = [C.c_int, C.c_void_p, C.c_void_p, C.c_void_p]
    return lib


def _smooth(n):
    for p in (2, 3, 5, 7):
        while n % p == 0:
            n //= p
    return n == 1


def test_no_plan_beyond_the_sums(lib):
    for n in range(513, 2049):
        assert lib.line_fft(n, None, None, None) == 0


def test_saturating_lines(lib):
    for n in (n for n in range(2, 513) if _smooth(n)):
        i = np.arange(n)
        below = np.nextafter(2.0, 1.0)  # the largest value of its binade
        faint = np.full(n, below * 2.0 ** -22 * (1 + 1j))  # counted as nothing
        faint[0] = below * (1 + 1j)
        for z in (np.full(n, below * (1 + 1j)), below * (1 + 1j) * np.where(i % 2, -1.0, 1.0),
                  below * np.sqrt(2.0) * np.exp(2j * np.pi * (i * (n // 3) % n) / n), faint):
            z = np.ascontiguousarray(z, dtype=np.complex128)
            out, most = np.empty_like(z), np.zeros(1)
            assert lib.line_fft(n, z.ctypes.data, out.ctypes.data, most.ctypes.data) == 1
            assert most[0] < 2.0 ** 62, n
            ref = np.fft.fft(z.astype(np.clongdouble))  # long double: numpy 2 keeps the precision
            scale = np.sqrt(np.sum(np.abs(ref) ** 2))
            # 3 units of 2^-53 in the 2-norm: a float64 FFT of these lengths has 1 to 2
            assert np.sqrt(np.sum(np.abs(out - ref) ** 2)) <= 3.4e-16 * scale, n
