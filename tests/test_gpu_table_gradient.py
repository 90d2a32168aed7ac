"""The table gradient with its moments in shared memory (one copy or several) and straight in
global memory: E_PP is linear in the table's values, so the gradient along any change of them is
the energy of that change."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import dftpy_gb300 as D
from dftpy_gb300 import synthetic as syn


@pytest.mark.parametrize("PME", [True, False])
@pytest.mark.parametrize("n,points", [(14, 12), (14, 4096), (48, 64), (48, 256), (40, 20001)])
def test_along_a_change(n, points, PME):
    lat = np.array([[8.0, 0.2, 0.0], [0.0, 9.0, 0.3], [0.5, 0.0, 10.0]])
    nr, rng = (n, n + 2, n - 1), np.random.default_rng(points)
    pos = rng.uniform(0, 1, (3, 3)) @ lat
    g = np.linspace(0.0, 40.0, points)
    change = rng.normal(size=points) / (1.0 + g)

    def pp(v):
        ions = D.Ions(symbols=["Al"] * 3, positions=pos, cell=lat)
        return D.LocalPseudo(grid=D.DirectGrid(lat, nr), ions=ions, PP_list={"Al": D.functional.RECPOT(r=g, v=v, zval=3)},
                             PME=PME)

    rho_np = syn.smooth_density(lat, nr, 9.0, seed=5, amp=0.5, kmax=1)
    a, b = pp(np.ones(points)), pp(change)
    grad = a.vloc_grad(D.DirectField(a.grid, data=rho_np))["Al"]
    energy = b(D.DirectField(b.grid, data=rho_np)).energy
    # sums of the same products in another order: within 1e-13 of their moduli, times a spline's condition
    assert abs(grad @ change - energy) <= 1e-12 * max(1.0, np.abs(grad * change).sum())
