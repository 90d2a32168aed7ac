"""The float64 evaluation on integer-pipe transforms against the numpy oracle: axis lengths
of one, two and three passes, odd row counts, partial tiles, the longest axis, and an axis
with a prime factor above 7 (the general path)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import dftpy_gb300 as D
from dftpy_gb300 import synthetic as syn
from oracle import ofdft_np as O

# the suite's float64 bars
E_RTOL, V_ATOL = 1e-10, 1e-9


@pytest.mark.parametrize("nr", [(2, 3, 4), (16, 15, 14), (27, 25, 21), (12, 125, 18), (18, 20, 512), (33, 16, 26)])
@pytest.mark.parametrize("kedf", ["TFVW", "WT", "WT-ab"])
def test_evaluation(nr, kedf):
    lat = np.array([[7.0, 0.3, 0.0], [0.0, 8.0, 0.5], [0.4, 0.0, 7.5]])
    rho_np = syn.smooth_density(lat, nr, 12.0, seed=5, amp=0.5, kmax=1)
    opts = dict(alpha=0.9, beta=0.7) if kedf == "WT-ab" else {}
    name = kedf[:2] if kedf.startswith("WT") else kedf
    grid = D.DirectGrid(lat, nr)
    total = D.TotalFunctional(KineticEnergyFunctional=D.Functional(type="KEDF", name=name, **opts),
                              XCFunctional=D.Functional(type="XC", name="LDA"), HARTREE=D.Functional(type="HARTREE"))
    rho = D.DirectField(grid, data=rho_np)
    og = O.Grid(lat, nr)
    ref = O.Total(og, O.make_terms(og, name, **opts))(rho_np)
    out = total(rho)
    assert abs(out.energy - ref["E"]) <= E_RTOL * max(1.0, abs(ref["E"]))
    assert float(np.abs(out.potential.numpy() - ref["V"]).max()) <= V_ATOL
    again = total(rho)  # the cached kernel, and the same bits
    assert again.energy == out.energy and np.array_equal(again.potential.numpy(), out.potential.numpy())
    only = total(rho, calcType={"E"})
    assert abs(only.energy - ref["E"]) <= E_RTOL * max(1.0, abs(ref["E"]))
