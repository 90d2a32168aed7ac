"""Which Ewald runs a caller pays for: the energy brings the forces along only where they share
the mesh (PME); with the exact structure factor they are a pass over the half grid per eight
atoms, and wait until they are asked for."""
import numpy as np
import pytest

import dftpy_gb300 as D
from dftpy_gb300.ewald import ewald


class Recorded(ewald):
    def _run(self, want_forces):
        self.runs = getattr(self, "runs", []) + [want_forces]
        self._parts = np.arange(4.0)
        if want_forces:
            self._forces = np.zeros((1, 3))


@pytest.mark.parametrize("PME,runs", [(False, [False, True]), (True, [True])])
def test_runs(PME, runs):
    lat = np.diag([8.0, 8.0, 8.0])
    ions = D.Ions(symbols=["Al"], positions=np.zeros((1, 3)), cell=lat)
    ew = Recorded(ions=ions, grid=D.DirectGrid(lat, (12, 12, 12)), PME=PME)
    ew.energy, ew.Energy_rec(), ew.Energy_corr()
    assert ew.runs == runs[:1] and (ew._forces is None) == (not runs[0])
    ew.forces, ew.energy
    assert ew.runs == runs
