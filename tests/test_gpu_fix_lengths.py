"""The float64 evaluation on integer-pipe transforms against the general path (library transforms),
close enough to see a few lost bits of the fixed-point scale: lengths of three passes on axis 0 (their
own buffers in the axis-0 kernels), lists of planes in parts on grids of few rows, nodes in many
shares.  An external potential of zero keeps an evaluation on the general path."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import dftpy_gb300 as D
from dftpy_gb300 import synthetic as syn
from dftpy_gb300.functional.external_potential import ExternalPotential

H = 0.4  # Bohr between points
U = 2.0 ** -53


def _case(nr):
    lat = np.diag([H * n for n in nr])
    rho_np = syn.smooth_density(lat, nr, 0.03 * H ** 3 * np.prod(nr), seed=5, amp=0.5, kmax=1)
    # The vW potential is the largest term: up to G^2/2 of the highest frequency times the rounding
    # of sqrt(rho)'s transform, over sqrt(rho).  A transform of up to nine radix passes with at most
    # four roundings each, forth and back, on either path: 144 U, taken once more for their sum.
    top = 0.5 * 3 * (np.pi / H) ** 2
    return D.DirectField(D.DirectGrid(lat, nr), data=rho_np), 144 * U * top * float(np.sqrt(rho_np.max() / rho_np.min()))


def _total(kedf, external=None, **kw):
    parts = dict(K=D.Functional(type="KEDF", name=kedf, **kw), X=D.Functional(type="XC", name="LDA"),
                 H=D.Functional(type="HARTREE"))
    if external is not None:
        parts["E"] = ExternalPotential(external)
    return D.TotalFunctional(**parts)


def _compare(out, ref, tol):
    assert abs(out.energy - ref.energy) <= 1e-13 * max(1.0, sum(abs(x) for x in ref.energies.values()))
    assert float(np.abs(out.potential.numpy() - ref.potential.numpy()).max()) <= tol


@pytest.mark.parametrize("nr", [(125, 6, 8), (162, 5, 6), (343, 4, 6), (486, 2, 3), (512, 4, 4), (6, 200, 8), (4, 4, 512)])
@pytest.mark.parametrize("kedf,kw", [("TFVW", {}), ("WT", {}), ("WT", dict(alpha=0.9, beta=0.7))])
def test_local_terms(nr, kedf, kw):
    rho, tol = _case(nr)
    zero = D.DirectField(rho.grid, data=np.zeros(nr))
    _compare(_total(kedf, **kw)(rho), _total(kedf, zero, **kw)(rho), tol)


@pytest.mark.parametrize("nr", [(125, 6, 8), (512, 4, 4), (128, 8, 8), (16, 16, 16), (4, 4, 512), (6, 200, 8)])
@pytest.mark.parametrize("kw", [dict(nsp=64, interp="hermite"), dict(nsp=64), dict(nsp=100, max_batch=7, kdd=1)])
def test_density_dependent_kernel(nr, kw):
    rho, tol = _case(nr)
    _compare(_total("LWT", **kw)(rho), _total("LWT", pipeline="cufft", **kw)(rho), tol)


@pytest.mark.parametrize("kedf,kw", [("TFVW", {}), ("WT", {}), ("LWT", dict(nsp=8)), ("LWT", dict(nsp=8, interp="hermite"))])
def test_nan_reaches_every_point(kedf, kw):
    nr = (16, 15, 18)
    rho_np = _case(nr)[0].numpy().copy()
    rho_np[3, 4, 5] = np.nan
    rho = D.DirectField(D.DirectGrid(np.diag([H * n for n in nr]), nr), data=rho_np)
    out = _total(kedf, **kw)(rho)
    assert np.isnan(out.energy) and np.isnan(out.potential.numpy()).all()


@pytest.mark.parametrize("kedf", ["TFVW", "WT"])
def test_infinity_reaches_every_point(kedf):
    nr = (16, 15, 18)
    rho_np = _case(nr)[0].numpy().copy()
    rho_np[3, 4, 5] = np.inf
    out = _total(kedf)(D.DirectField(D.DirectGrid(np.diag([H * n for n in nr]), nr), data=rho_np))
    assert not np.isfinite(out.energy) and not np.isfinite(out.potential.numpy()).any()
