"""|G|^2 of the float64 evaluation in a cell whose reciprocal vectors nearly cancel: the Hartree
potential of one plane wave is 4 pi / |G|^2 times the wave, with |G|^2 in rational arithmetic."""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import dftpy_gb300 as D

LAT = [[10.0, 0.0, 0.0], [9.95, 0.5, 0.0], [9.95, 0.25, 0.5]]
N = 64
U = 2.0 ** -53


def reciprocal():
    """2 pi inv(LAT)^T, operation by operation as the grid forms it."""
    (a0, a1, a2), (a3, a4, a5), (a6, a7, a8) = LAT
    det = a0 * (a4 * a8 - a5 * a7) - a1 * (a3 * a8 - a5 * a6) + a2 * (a3 * a7 - a4 * a6)
    inv = [[(a4 * a8 - a5 * a7) / det, (a2 * a7 - a1 * a8) / det, (a1 * a5 - a2 * a4) / det],
           [(a5 * a6 - a3 * a8) / det, (a0 * a8 - a2 * a6) / det, (a2 * a3 - a0 * a5) / det],
           [(a3 * a7 - a4 * a6) / det, (a1 * a6 - a0 * a7) / det, (a0 * a4 - a1 * a3) / det]]
    return [[2.0 * np.pi * inv[k][j] for k in range(3)] for j in range(3)]


@pytest.mark.parametrize("wave", [(3, 3, 3), (9, 9, 9), (23, 24, 24), (29, 28, 26), (5, -4, 7)])
def test_one_plane_wave(wave):
    b = reciprocal()
    g = [sum(Fraction(f) * Fraction(b[d][c]) for d, f in enumerate(wave)) for c in range(3)]
    gg = float(sum(x * x for x in g))
    # a component is three products and two sums of terms f_d b_dc, so within 3 U of their moduli
    terms = [sum(abs(f * b[d][c]) for d, f in enumerate(wave)) for c in range(3)]
    bound = 2.0 * sum(abs(float(x)) * 3 * U * t for x, t in zip(g, terms)) / gg
    bound += 16 * U  # squares and their sum 3, reciprocal and factor 4, the wave's own rounding and six passes 9
    i = np.arange(N)
    phase = (wave[0] * i[:, None, None] + wave[1] * i[None, :, None] + wave[2] * i[None, None, :]) % N
    cos = np.cos(2.0 * np.pi * np.arange(N) / N)[phase]
    rho = D.DirectField(D.DirectGrid(np.array(LAT), (N, N, N)), data=cos)
    V = D.Functional(type="HARTREE")(rho).potential.numpy()
    got = float((V * cos).sum() / (cos * cos).sum())
    assert abs(got * gg / (4.0 * np.pi) - 1.0) <= bound
