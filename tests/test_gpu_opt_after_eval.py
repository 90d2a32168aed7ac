"""An optimisation does not depend on an evaluation that came before it: the bits are the same
(the optimiser and a single evaluation are two implementations, whose kernels and sums differ in
the last bits)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import dftpy_gb300 as D
from dftpy_gb300 import synthetic as syn


@pytest.mark.parametrize("opts", [{}, dict(alpha=0.9, beta=0.7)])
def test_same_bits_with_and_without_an_evaluation(opts):
    lat, pos = syn.fcc_cell(7.6)
    nr = (24, 20, 18)
    rho_np = syn.smooth_density(lat, nr, 12.0, seed=2, amp=0.4)
    g, v = syn.analytic_vloc(3.0, 1.0)

    def solve(evaluate):
        grid = D.DirectGrid(lat, nr)
        pp = D.LocalPseudo(grid=grid, ions=D.Ions(symbols=["Al"] * 4, positions=pos, cell=lat),
                           PP_list={"Al": D.functional.RECPOT(r=g, v=v, zval=3)}, PME=True)
        total = D.TotalFunctional(KE=D.Functional(type="KEDF", name="WT", **opts), XC=D.Functional(type="XC", name="LDA"),
                                  HARTREE=D.Functional(type="HARTREE"), PSEUDO=pp)
        rho = D.DirectField(grid, data=rho_np)
        if evaluate:
            total(rho)
        opt = D.Optimization(optimization_method="LBFGS", EnergyEvaluator=total,
                             optimization_options={"maxiter": 6, "econv": 1e-14})
        out = opt.optimize_rho(guess_rho=rho)
        after = total(rho) if evaluate else None
        return out.numpy(), opt.functional.energy, after

    (a, ea, after), (b, eb, _) = solve(True), solve(False)
    assert ea == eb and np.array_equal(a, b)
    assert after is not None and np.isfinite(after.energy)
