"""Public settings of a local pseudopotential that change between two moves of the ions: the
potential and the forces of the new geometry take them, as a pseudopotential made anew does."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import dftpy_gb300 as D
from dftpy_gb300 import synthetic as syn

LAT, POS = syn.fcc_cell(7.6)
NR = (24, 20, 18)


def _pp(pos, v, PME=True, order=10, nr=NR):
    g = syn.analytic_vloc(3.0, 1.0)[0]
    return D.LocalPseudo(grid=D.DirectGrid(LAT, nr), ions=D.Ions(symbols=["Al"] * 4, positions=pos, cell=LAT),
                         PP_list={"Al": D.functional.RECPOT(r=g, v=v, zval=3)}, PME=PME, BsplineOrder=order)


@pytest.mark.parametrize("what", ["PME", "BsplineOrder", "table in place", "readpp"])
def test_set_positions_takes_them(what):
    rng = np.random.default_rng(1)
    v = syn.analytic_vloc(3.0, 1.0)[1]
    moved = POS + rng.normal(0, 0.2, POS.shape)
    rho_np = syn.smooth_density(LAT, NR, 12.0, seed=2, amp=0.4)
    pp = _pp(POS, v.copy())
    pp.vreal
    kw = {}
    if what == "PME":
        pp.PME = kw["PME"] = False
    elif what == "BsplineOrder":
        pp.BsplineOrder = kw["order"] = 6
    elif what == "table in place":
        pp.readpp.vp["Al"][1:] *= 1.125
        v = v.copy()
        v[1:] *= 1.125
    else:
        v = 1.125 * v
        pp.readpp = _pp(POS, v).readpp
    pp.set_positions(moved)
    ref = _pp(moved, v, **kw)
    assert np.array_equal(pp.vreal.numpy(), ref.vreal.numpy())
    rho = lambda p: D.DirectField(p.grid, data=rho_np)
    assert np.allclose(pp.forces(rho(pp)), ref.forces(rho(ref)), rtol=0, atol=1e-13)
