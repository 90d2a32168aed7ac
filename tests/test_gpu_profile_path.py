"""Profiling times the evaluation that runs without it: the same bits, the same launches, and a time
for every class of kernel that it has."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

import dftpy_gb300 as D
from dftpy_gb300 import _lib, synthetic as syn


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("kedf,kw", [("TFVW", {}), ("WT", {}), ("LWT", dict(nsp=8)), ("LWT", dict(nsp=8, interp="hermite"))])
def test_same_bits(kedf, kw, dtype):
    nr = (32, 32, 32)
    lat = np.diag([9.0, 9.0, 9.0])
    grid = D.DirectGrid(lat, nr)
    rho = D.DirectField(grid, data=syn.smooth_density(lat, nr, 20.0, seed=5, amp=0.5, kmax=1), dtype=dtype)
    total = D.TotalFunctional(K=D.Functional(type="KEDF", name=kedf, **kw), X=D.Functional(type="XC", name="LDA"),
                              H=D.Functional(type="HARTREE"))
    plain = total(rho)
    ev, lib = total.evaluator(grid, dtype), _lib.load()
    launches = ev.stats()[1]
    _lib.check(lib.ofdft_eval_profile(ev.h, 1))
    out = total(rho)
    ms, by, la, n = (C.c_double * 16)(), (C.c_double * 16)(), (C.c_longlong * 16)(), C.c_int()
    _lib.check(lib.ofdft_eval_profile_read(ev.h, 16, ms, by, la, C.byref(n)))
    _lib.check(lib.ofdft_eval_profile(ev.h, 0))
    names = {lib.ofdft_profile_class_name(i).decode(): i for i in range(n.value)}
    assert out.energy == plain.energy and torch.equal(out.potential, plain.potential)
    assert ev.stats()[1] == launches
    want = {"prepass", "postpass", "reduce", "fix_fft" if dtype == torch.float64 else "cufft"}
    if kedf == "LWT":
        want |= {"lwt_nodes", "lwt_interp", "lwt_pot2", "fz_axis1", "fz_hat"}
    assert want <= {k for k, i in names.items() if la[i] > 0 and ms[i] > 0 and by[i] > 0}
    assert dtype == torch.float32 or la[names["cufft"]] == 0
