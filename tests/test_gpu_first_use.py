"""The first use of a mechanism's own kernels by calls that can do without them (source terms, the per-state update):
while another stream is captured, by several threads at once, and when loading them fails for a reason that passes (a damaged file in the cache of
compiled kernels stands for one), after which the next call loads them."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT, mech

pytestmark = pytest.mark.gpu


def _cells(torch, rc, n=300):
    from gdtk_gb300.workloads import h2air_cells
    T, p, Y = h2air_cells(rc.species_names, rc.mol_masses, n, seed=12, gas_file=rc.gmodel.file_name)
    T, p, Y = (torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda") for a in (T, p, Y))
    rho, _ = rc.thermo_from_pT(p, T, Y)
    return rho, T, Y


def _loaded(rc):
    from gdtk_gb300 import lib
    return lib().chem_reactor_update_cells_noalloc(rc.reactor.id, 0, *[None] * 7, 1.0, 0.0, 3, None) == 0   # which needs them loaded


def test_source_terms_while_another_stream_is_captured():
    import torch
    from gdtk_gb300 import check, lib
    from gdtk_gb300.cells import ReactorCells
    rc = ReactorCells(mech("j92-gas.lua"), mech("j92-chem.lua"))
    rho, T, Y = _cells(torch, rc)
    out, x = torch.empty_like(Y), torch.zeros(8, device="cuda")
    other = torch.cuda.Stream()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    vp = lambda t: ctypes.c_void_p(t.data_ptr())
    with torch.cuda.graph(graph, capture_error_mode="global"):
        x += 1.0
        check(lib().chem_reactor_source_terms_cells(rc.reactor.id, rho.shape[0], vp(rho), vp(T), vp(Y), vp(out), None,
                                                    ctypes.c_void_p(other.cuda_stream)), "source terms")
        x += 1.0
    assert _loaded(rc)
    graph.replay()
    torch.cuda.synchronize()
    assert bool((x == 2.0).all())
    assert torch.equal(out, rc.source_terms(rho, T, Y))


def test_source_terms_by_several_threads():
    import threading
    import torch
    from gdtk_gb300 import lib
    from gdtk_gb300.cells import ReactorCells
    vp = lambda t: ctypes.c_void_p(t.data_ptr())
    for name in ("j92", "j92", "j92"):   # a fresh reactor each time
        rc = ReactorCells(mech(name + "-gas.lua"), mech(name + "-chem.lua"))
        rho, T, Y = _cells(torch, rc)
        n = 6
        outs, streams, rcs = [torch.empty_like(Y) for _ in range(n)], [torch.cuda.Stream() for _ in range(n)], [None] * n
        torch.cuda.synchronize()
        gate = threading.Barrier(n)

        def call(k):
            gate.wait()
            for _ in range(20):
                rcs[k] = lib().chem_reactor_source_terms_cells(rc.reactor.id, rho.shape[0], vp(rho), vp(T), vp(Y), vp(outs[k]), None,
                                                               ctypes.c_void_p(streams[k].cuda_stream))
        threads = [threading.Thread(target=call, args=(k,)) for k in range(n)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        torch.cuda.synchronize()
        assert rcs == [0] * n
        want = rc.source_terms(rho, T, Y)
        for out in outs:
            assert torch.equal(out, want)


CHILD = """
import os, sys
import torch
sys.path.insert(0, %r); sys.path.insert(0, %r)
import test_gpu_first_use as t
from conftest import mech
from gdtk_gb300 import lib
from gdtk_gb300.cells import ReactorCells
from gdtk_gb300.gas import GasState
rc = ReactorCells(mech("j92-gas.lua"), mech("j92-chem.lua"))
rho, T, Y = t._cells(torch, rc)
def state():
    gs = GasState(rc.gmodel)
    gs.p, gs.T, gs.massf = 1.0e5, 1500.0, [0.7, 0.2, 0.05] + [0.05 / 10] * 10
    gs.update_thermo_from_pT()
    rc.reactor.update_state(gs, 1.0e-7)
    return gs.T
if sys.argv[1] == "make":
    rc.source_terms(rho, T, Y)
    assert t._loaded(rc)
else:
    path, = [os.path.join(sys.argv[2], f) for f in os.listdir(sys.argv[2]) if f.endswith(".cubin")]
    good = open(path, "rb").read()
    open(path, "wb").write(b"not a compiled kernel\\n" * 20)
    a, s = rc.source_terms(rho, T, Y), state()
    assert b"cuModuleLoadData" in lib().gdtk_last_error() and not t._loaded(rc)
    open(path, "wb").write(good)
    b = rc.source_terms(rho, T, Y)
    assert t._loaded(rc)
    assert abs(state() - s) <= 1e-7 * s
    assert ((a - b).abs().amax(dim=1) <= 1e-10 * a.abs().amax(dim=1) + 1e-30).all()
"""


def test_a_failure_that_passes(tmp_path):
    env = dict(os.environ, GDTK_JIT_CACHE=str(tmp_path))
    for what in ("make", "use"):
        r = subprocess.run([sys.executable, "-c", CHILD % (ROOT, os.path.join(ROOT, "tests")), what, str(tmp_path)], env=env,
                           capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr
