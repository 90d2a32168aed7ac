"""v_loc inside a CUDA graph capture (after one call outside, which sizes its buffers), and moved
ions while a captured call may still be running."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

import dftpy_gb300 as D
from dftpy_gb300 import _lib, synthetic as syn


@pytest.mark.parametrize("PME", [True, False])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_capture_and_replay(PME, dtype):
    lat, pos = syn.fcc_cell(7.6)
    nr = (24, 20, 18)
    g, v = syn.analytic_vloc(3.0, 1.0)

    def make(p):
        return D.LocalPseudo(grid=D.DirectGrid(lat, nr), ions=D.Ions(symbols=["Al"] * 4, positions=p, cell=lat),
                             PP_list={"Al": D.functional.RECPOT(r=g, v=v, zval=3)}, PME=PME)

    pp, lib = make(pos), _lib.load()
    ref = pp.vreal_for(dtype).as_subclass(torch.Tensor).clone()
    out = torch.zeros(nr, dtype=dtype, device="cuda")
    h = pp._handle(dtype)
    torch.cuda.synchronize()
    st, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=st):
        rc = lib.ofdft_pseudo_vloc(h, C.c_void_p(out.data_ptr()), C.c_void_p(st.cuda_stream))
    assert rc == _lib.OK
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, ref)
    # a call outside the capture, on another stream, after the graph
    assert torch.equal(pp.vreal_for(dtype).as_subclass(torch.Tensor), ref)
    moved = pos + np.random.default_rng(4).normal(0, 0.2, pos.shape)
    graph.replay()
    pp.set_positions(moved)  # waits for the replay
    assert torch.equal(out, ref)
    assert torch.equal(pp.vreal_for(dtype).as_subclass(torch.Tensor),
                       make(moved).vreal_for(dtype).as_subclass(torch.Tensor))


@pytest.mark.parametrize("PME", [True, False])
def test_moved_ions_beside_another_stream(PME):
    """Ions moved while a call on another stream may still run, and a call on a third stream after it."""
    lat, pos = syn.fcc_cell(7.6)
    nr = (48, 40, 36)
    g, v = syn.analytic_vloc(3.0, 1.0)
    rng = np.random.default_rng(5)
    moves = [pos + rng.normal(0, 0.2, pos.shape) for _ in range(6)]

    def make(p):
        return D.LocalPseudo(grid=D.DirectGrid(lat, nr), ions=D.Ions(symbols=["Al"] * 4, positions=p, cell=lat),
                             PP_list={"Al": D.functional.RECPOT(r=g, v=v, zval=3)}, PME=PME)

    want = [make(p).vreal.as_subclass(torch.Tensor) for p in moves]
    torch.cuda.synchronize()
    pp, streams, got = make(pos), [torch.cuda.Stream() for _ in range(3)], []
    for i, p in enumerate(moves):
        pp.set_positions(p)
        with torch.cuda.stream(streams[i % 3]):
            got.append(pp.vreal.as_subclass(torch.Tensor))
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, want))
