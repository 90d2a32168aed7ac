"""The integer-pipe line transforms (csrc/fix_fft.cuh), run on the host: every length the
plans take against numpy's long double DFT, on lines that stress the scale (flat, decaying,
one dominant element, coherent sums whose outputs reach the 1-norm, tiny and huge values)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include "fix_fft.cuh"
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
extern "C" int line_fft(int n, const double* in, double* out) {  // 0 when n has no plan
    Plan p;
    if (!plan_radices(n, p)) return 0;
    std::vector<I2> a(n), b(n);
    std::vector<Tw> tw(n);
    for (int k = 0; k < n; ++k) {
        const long double t = -2.0L * 3.14159265358979323846264338327950288L * k / n;
        tw[k] = tw_of((long long)std::llroundl(std::cos(t) * (long double)kOne),
                      (long long)std::llroundl(std::sin(t) * (long double)kOne));
    }
    int em = 0;
    for (int i = 0; i < 2 * n; ++i) em = std::max(em, expo(in[i]));
    unsigned most = 0, sum = 0;
    for (int j = 0; j < n / p.r[0]; ++j) {
        unsigned s = 2 * p.r[0];
        for (int q = 0; q < p.r[0]; ++q) {
            const double* v = in + 2 * (j + q * (n / p.r[0]));
            s += bound(expo(v[0]), em) + bound(expo(v[1]), em);
        }
        most = std::max(most, s);
        sum += s;
    }
    const Scale c{em, 32 - __builtin_clz(most)};
    const int ds = p.np > 1 ? 32 - __builtin_clz(sum) - c.sh : 0;
    const int k = fix_shift(c);
    for (int i = 0; i < n; ++i) a[i] = I2{to_fix(in[2 * i], k), to_fix(in[2 * i + 1], k)};
    int Ns = 1;
    for (int q = 0; q < p.np; ++q) {
        const int R = p.r[q], m = n / R, step = n / (Ns * R);
        for (int j = 0; j < m; ++j) {
            const int k = j % Ns;
            I2 u[16];
            for (int r = 0; r < R; ++r) {
                u[r] = a[j + r * m];
                if (r && q) u[r] = cmul(u[r], tw[k * r * step]);
                if (q) {
                    const int d = pass_shift(ds, q, p.np, p.r[1]);
                    u[r] = I2{shr(u[r].x, d), shr(u[r].y, d)};
                }
            }
            dft(R, u);
            for (int r = 0; r < R; ++r) b[(j / Ns) * Ns * R + k + r * Ns] = u[r];
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
    d = tmp_path_factory.mktemp("fix")
    src = d / "line.cpp"
    src.write_text(SRC)
    so = d / "line.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I/usr/local/cuda/include",
                    "-I" + os.path.join(REPO, "dftpy_gb300", "csrc"), "-o", str(so), str(src)], check=True)
    lib = C.CDLL(str(so))
    lib.line_fft.argtypes = [C.c_int, C.c_void_p, C.c_void_p]
    return lib


def _smooth(n):
    for p in (2, 3, 5, 7):
        while n % p == 0:
            n //= p
    return n == 1


def _lines(n, rng):
    i = np.arange(n)
    z = rng.normal(size=n) + 1j * rng.normal(size=n)
    wave = np.exp(2j * np.pi * (i * (n // 3) % n) / n)
    return [z, z * np.exp(-0.3 * i), np.where(i == n // 3, z, 1e-9 * z), np.full(n, 1.0 + 1.0j), wave,
            np.where(i % 2 == 0, 1.0, -1.0) + 0j, z * 1e-200, z * 1e200, np.zeros(n, complex)]


def test_lengths(lib):
    rng = np.random.default_rng(0)
    for n in range(2, 513):
        if not _smooth(n):
            assert lib.line_fft(n, None, None) == 0
            continue
        if n > 128 and n % 5 and n % 16 and n not in (343, 486):
            continue  # enough of the long ones
        k = np.arange(n)
        w = -2 * np.longdouble("3.14159265358979323846264338327950288") * (np.outer(k, k) % n).astype(np.longdouble) / n
        F = np.cos(w) + 1j * np.sin(w)
        for z in _lines(n, rng):
            z = np.ascontiguousarray(z, dtype=np.complex128)
            out = np.empty_like(z)
            assert lib.line_fft(n, z.ctypes.data, out.ctypes.data) == 1
            ref = F @ z.astype(np.clongdouble)
            # 3 units of 2^-53 in the 2-norm: a float64 FFT of these lengths has 1 to 2
            scale = np.sqrt(np.sum(np.abs(ref) ** 2))
            assert np.sqrt(np.sum(np.abs(out - ref) ** 2)) <= 3.4e-16 * scale, (n, scale)


def test_nonfinite(lib):
    for bad in (np.inf, np.nan):
        z = np.ones(24, complex)
        z[5] = bad
        out = np.empty_like(z)
        lib.line_fft(24, z.ctypes.data, out.ctypes.data)
        assert np.isnan(out.real).all()
