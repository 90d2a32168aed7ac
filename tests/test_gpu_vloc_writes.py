"""A write to v_loc that PyTorch's version counter does not see, or a potential put into the
evaluator's handle directly, against what the next call uses."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

import dftpy_gb300 as D
from dftpy_gb300 import _lib, synthetic as syn


def test_every_write_reaches_the_next_call():
    lat, pos = syn.fcc_cell(7.6)
    nr = (24, 20, 18)
    g, v = syn.analytic_vloc(3.0, 1.0)
    grid = D.DirectGrid(lat, nr)
    pp = D.LocalPseudo(grid=grid, ions=D.Ions(symbols=["Al"] * 4, positions=pos, cell=lat),
                       PP_list={"Al": D.functional.RECPOT(r=g, v=v, zval=3)}, PME=True)
    total = D.TotalFunctional(KE=D.Functional(type="KEDF", name="TFVW"), HARTREE=D.Functional(type="HARTREE"), PSEUDO=pp)
    rho = D.DirectField(grid, data=syn.smooth_density(lat, nr, 12.0, seed=2, amp=0.4))
    E0 = total(rho).energy
    writes = [lambda t: t.data.add_(0.5), lambda t: torch.from_dlpack(t.as_subclass(torch.Tensor).detach()).add_(0.5)]
    for n, write in enumerate(writes, 1):
        write(pp.vreal)
        assert abs(total(rho).energy - E0 - 0.5 * n * 12.0) < 1e-9, n
    E1 = total(rho).energy
    ev = total.evaluator(grid, torch.float64)
    zero = torch.zeros(nr, dtype=torch.float64, device="cuda")
    _lib.check(_lib.load().ofdft_eval_set_vloc(ev.h, C.c_void_p(zero.data_ptr()),
                                               C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    assert total(rho).energy == E1
