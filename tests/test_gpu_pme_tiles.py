"""Particle-mesh spreading against the numpy oracle where its 8 x 8 x 32 tiles end: a last axis
shorter than a tile, a partial second tile, an odd length, whole tiles, and an atom whose stencil
wraps around every axis."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import dftpy_gb300 as D
from dftpy_gb300 import synthetic as syn
from oracle import ofdft_np as O

# the suite's float64 bars
E_RTOL, V_ATOL = 1e-10, 1e-9


@pytest.mark.parametrize("nr", [(20, 24, 22), (14, 18, 40), (13, 16, 33), (16, 12, 64)])
def test_local_potential_and_ewald(nr):
    lat = np.array([[8.0, 0.2, 0.0], [0.0, 9.0, 0.3], [0.5, 0.0, 10.0]])
    frac = np.array([[0.999, 0.999, 0.999], [0.5, 0.02, 0.49], [0.27, 0.51, 0.76]])
    pos = frac @ lat
    gp, vp = syn.analytic_vloc(3.0, 1.0)
    grid = D.DirectGrid(lat, nr)
    ions = D.Ions(symbols=["Al"] * len(pos), positions=pos, cell=lat)
    pp = D.LocalPseudo(grid=grid, ions=ions, PP_list={"Al": D.functional.RECPOT(r=gp, v=vp, zval=3)}, PME=True)
    rho_np = syn.smooth_density(lat, nr, 9.0, seed=5, amp=0.5, kmax=1)
    og = O.Grid(lat, nr)
    ref = O.LocalPseudo(og, pos, np.zeros(len(pos), dtype=int), [(gp, vp)], PME=True)(rho_np, ("E", "V"))
    out = pp(D.DirectField(grid, data=rho_np))
    assert abs(out.energy - ref["E"]) <= E_RTOL * max(len(pos), abs(ref["E"]))
    assert float(np.abs(out.potential.numpy() - ref["V"]).max()) <= V_ATOL
    ew, oew = pp.get_ewald(), O.Ewald(og, pos, np.full(len(pos), 3.0), PME=True)
    assert abs(ew.energy - oew.energy()) <= E_RTOL * max(len(pos), abs(oew.energy()))


@pytest.mark.parametrize("nr", [(20, 12, 34), (17, 13, 16)])  # a partial slab of four points, of one
def test_many_atoms(nr):
    """From 4096 atoms on the tiles take their atoms from lists of the slabs along axis 0."""
    lat = np.array([[8.0, 0.2, 0.0], [0.0, 9.0, 0.3], [0.5, 0.0, 10.0]])
    pos = np.random.default_rng(7).uniform(0, 1, (4100, 3)) @ lat
    gp, vp = syn.analytic_vloc(3.0, 1.0)
    grid = D.DirectGrid(lat, nr)
    ions = D.Ions(symbols=["Al"] * len(pos), positions=pos, cell=lat)
    pp = D.LocalPseudo(grid=grid, ions=ions, PP_list={"Al": D.functional.RECPOT(r=gp, v=vp, zval=3)}, PME=True)
    og = O.Grid(lat, nr)
    rho_np = syn.smooth_density(lat, nr, 9.0, seed=5, amp=0.5, kmax=1)
    ref = O.LocalPseudo(og, pos, np.zeros(len(pos), dtype=int), [(gp, vp)], PME=True)(rho_np, ("E", "V"))
    out = pp(D.DirectField(grid, data=rho_np))
    assert abs(out.energy - ref["E"]) <= E_RTOL * max(len(pos), abs(ref["E"]))
    # a potential that grows with the atoms: the bar is relative to its range
    assert float(np.abs(out.potential.numpy() - ref["V"]).max()) <= V_ATOL * max(1.0, float(np.abs(ref["V"]).max()))
    again = pp.vreal.numpy().copy()
    pp.set_positions(pos)
    assert np.array_equal(pp.vreal.numpy(), again)
