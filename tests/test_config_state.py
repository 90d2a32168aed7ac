"""What a call must notice about its functionals although their native configuration is kept:
a class or an object with a ``configure`` or ``engines`` of its own, option values that change
their type, and options that cannot be copied."""
import threading

import numpy as np
import pytest

import dftpy_gb300 as D
from dftpy_gb300 import _lib
from dftpy_gb300.functional.kedf import KEDF
from dftpy_gb300.functional.semilocal import XC

try:
    _lib.load()
except Exception:  # not built here
    pytestmark = pytest.mark.skip(reason="native library not built")


class ScaledTF(KEDF):
    factor = 1.0

    def configure(self, cfg, engines=None):
        KEDF.configure(self, cfg, engines)
        cfg.tf_x = self.factor


class Switched(KEDF):
    which = ("TF",)

    def engines(self, name=None):
        return self.which


class NoXC(XC):
    on = 1

    def configure(self, cfg):
        cfg.xc_lda = self.on


def _cfg(total):
    return total._config().cfg


def test_subclasses():
    ke, sw, xc = ScaledTF(name="TF"), Switched(name="TF"), NoXC(name="LDA")
    t1, t2 = D.TotalFunctional(KE=ke, XC=xc), D.TotalFunctional(KE=sw)
    assert _cfg(t1).tf_x == 1.0 and _cfg(t1).xc_lda == 1 and _cfg(t2).kedf_terms == _lib.KE_TF
    ke.factor, xc.on, sw.which = 0.5, 0, ("VW",)
    assert _cfg(t1).tf_x == 0.5 and _cfg(t1).xc_lda == 0 and _cfg(t2).kedf_terms == _lib.KE_VW


def test_replaced_methods(monkeypatch):
    ke = D.Functional(type="KEDF", name="TF")
    total = D.TotalFunctional(KE=ke)
    assert _cfg(total).tf_x == 1.0
    plain = ke.configure

    def mine(cfg, engines=None):
        plain(cfg, engines)
        cfg.tf_x = 0.25
    ke.configure = mine
    assert _cfg(total).tf_x == 0.25
    del ke.configure
    assert _cfg(total).tf_x == 1.0
    original = KEDF.configure

    def patched(self, cfg, engines=None):
        original(self, cfg, engines)
        cfg.tf_x = 0.75
    monkeypatch.setattr(KEDF, "configure", patched)
    assert _cfg(total).tf_x == 0.75


def test_option_values():
    ke = D.Functional(type="KEDF", name="GGA", k_str="LKT", gga_remove_vw=2)
    total = D.TotalFunctional(KE=ke)
    assert _cfg(total).gga_remove_vw == 2.0
    ke.options["gga_remove_vw"] = np.int64(2)  # not a Python number: counts as "on"
    assert _cfg(total).gga_remove_vw == 1.0
    ke.options["note"] = threading.Lock()  # cannot be copied
    ke.options["x"] = 0.5
    assert _cfg(total).tf_x == 0.5
    ke.options["x"] = 0.6
    assert _cfg(total).tf_x == 0.6


def test_overridden_evaluator():
    """An evaluator() or _fusable() of a derived class is asked on every evaluation."""
    asked = []

    class Mine(D.TotalFunctional):
        def evaluator(self, grid, dtype):
            asked.append("evaluator")
            raise RuntimeError("mine")

    class Always(D.TotalFunctional):
        def _fusable(self):
            return True

        def _evaluator(self, c, grid, dtype):
            asked.append(c.key is not None)
            raise RuntimeError("mine")

    lat = np.diag([8.0, 8.0, 8.0])
    rho = D.DirectField(D.DirectGrid(lat, (6, 6, 6)), data=np.full((6, 6, 6), 0.03), device="cpu")
    for cls in (Mine, Always):
        total = cls(KE=D.Functional(type="KEDF", name="TF"))
        for _ in range(2):
            with pytest.raises(RuntimeError, match="mine"):
                total(rho)
    assert asked == ["evaluator", "evaluator", True, True]
