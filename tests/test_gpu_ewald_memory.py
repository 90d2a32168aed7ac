"""What an Ewald sum keeps on the device after it: its meshes up to a bound, nothing of them
above (320^3 points: 262 MB each)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

import dftpy_gb300 as D
from dftpy_gb300.ewald import ewald


def _held(n, PME):
    lat = np.diag([0.25 * n] * 3)
    grid = D.DirectGrid(lat, (n, n, n))
    pos = np.random.default_rng(0).uniform(0, 0.25 * n, (4, 3))
    ions = D.Ions(symbols=["Al"] * 4, positions=pos, cell=lat)
    ions.set_charges({"Al": 3.0})
    D.DirectField(grid, data=np.zeros((n, n, n))).fft()  # the transform's plan is the grid's, not the sum's
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    ew = ewald(ions=ions, grid=grid, PME=PME)
    ew.energy, ew.forces, ew.stress
    torch.cuda.synchronize()
    return before - torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("PME", [True, False])
def test_large_meshes_are_given_back(PME):
    _held(24, PME)  # loads the kernels
    assert _held(320, PME) < 64 << 20


def test_a_kept_mesh_is_bounded():
    _held(24, True)
    assert _held(200, True) < 3 * 8 * 200 ** 3  # two meshes of N doubles and the plans' tables
