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


@pytest.mark.parametrize("nr", [(11, 13, 2), (22, 23, 26)])  # one block of the sums; a partial last one
@pytest.mark.parametrize("kedf", ["TFVW", "WT", "WT-ab"])
def test_general_path_in_split_passes(nr, kedf):
    test_evaluation(nr, kedf)


@pytest.mark.parametrize("nr,opts", [
    ((2, 3, 4), dict(nsp=3)),
    ((16, 15, 14), dict(nsp=8, max_batch=3)),  # several batches of nodes, the last one short
    ((16, 15, 14), dict(nsp=8, kfmin=0.8, kfmax=2.0, interp="hermite")),  # points below the first node
    ((16, 15, 14), dict(nsp=8, kfmax=1.2)),  # points above the last one
    ((33, 16, 26), dict(ratio=1.15)),  # an odd number of rows; a prime factor of 11 or 13: the general path
    ((25, 27, 21), dict(nsp=16, interp="hermite")),  # an odd number of rows
    ((12, 125, 18), dict(nsp=5, kdd=1)),
    ((12, 125, 18), dict(nsp=5, kdd=2, interp="hermite")),
    ((18, 20, 512), dict(nsp=4)),
    ((32, 30, 36), dict(nsp=64, alpha=1.2, beta=0.5)),
])
def test_density_dependent_kernel(nr, opts):
    lat = np.array([[7.0, 0.3, 0.0], [0.0, 8.0, 0.5], [0.4, 0.0, 7.5]])
    rho_np = syn.smooth_density(lat, nr, 12.0, seed=5, amp=0.5, kmax=1)
    total = D.TotalFunctional(KineticEnergyFunctional=D.Functional(type="KEDF", name="LWT", **opts),
                              XCFunctional=D.Functional(type="XC", name="LDA"), HARTREE=D.Functional(type="HARTREE"))
    rho = D.DirectField(D.DirectGrid(lat, nr), data=rho_np)
    og = O.Grid(lat, nr)
    terms = O.make_terms(og, "LWT", **{k: v for k, v in opts.items() if k != "max_batch"})
    ref = O.Total(og, terms)(rho_np)
    out = total(rho)
    assert abs(out.energy - ref["E"]) <= E_RTOL * max(1.0, abs(ref["E"]))
    assert float(np.abs(out.potential.numpy() - ref["V"]).max()) <= V_ATOL
    again = total(rho)
    assert again.energy == out.energy and np.array_equal(again.potential.numpy(), out.potential.numpy())
    only = total(rho, calcType={"E"})
    assert abs(only.energy - ref["E"]) <= E_RTOL * max(1.0, abs(ref["E"]))


def test_density_dependent_kernel_of_a_molecule():
    """Vacuum and a negative value: k_F below the first node, and one point at the last node,
    inside the last interval or outside every one by k_F's last bit (numpy's cube root has
    another one there, so the general path is the reference)."""
    nr, lat = (16, 18, 20), np.diag([9.0, 8.0, 10.0])
    grid = D.DirectGrid(lat, nr)
    x = np.stack(np.meshgrid(*[(np.arange(n) / n - 0.5) * a for n, a in zip(nr, np.diag(lat))], indexing="ij"))
    rho_np = 0.26 * np.exp(-0.7 * ((x - 0.1) ** 2).sum(0))
    rho_np[0, 0, 0] = -1e-5
    rho = D.DirectField(grid, data=rho_np)
    for interp in ("linear", "hermite"):
        kw = dict(type="KEDF", name="LWT-NL", nsp=16, interp=interp)
        out, ref = D.Functional(**kw)(rho), D.Functional(pipeline="cufft", **kw)(rho)
        assert abs(out.energy - ref.energy) <= E_RTOL * max(1.0, abs(ref.energy))
        assert float(np.abs(out.potential.numpy() - ref.potential.numpy()).max()) <= V_ATOL
