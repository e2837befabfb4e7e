"""The kernel with a group of lanes per cell against the one-thread-per-cell kernel, bit for bit.

The library picks 4, 8, 16 or 32 lanes per cell, or one thread, from the batch's size; no cell's result
may depend on that.  chem_reactor_configure with a block size asks for the one-thread-per-cell kernel, so a
configured reactor is the reference.  The sizes lie around one warp's cells (32 / L), around the sizes where
the choice changes, and include batches whose tail is regrouped.
"""
import ctypes

import numpy as np
import pytest

from conftest import mech

pytestmark = pytest.mark.gpu

# mechanism, T range, interval: RKF (given and equilibrium backward rates), alpha-QSS tight, falloff rates
MECHS = {"park5": (2000.0, 8000.0, 2.0e-7), "gupta5": (2000.0, 6000.0, 1.0e-7), "n2": (3000.0, 6000.0, 1.0e-6),
         "j92": (400.0, 2600.0, 2.0e-7), "stanford": (1000.0, 2400.0, 1.0e-7), "drm19": (1000.0, 2400.0, 1.0e-7),
         "h2o2forms": (900.0, 2400.0, 1.0e-7)}
SIZES = {"park5": (1, 3, 1025, 2051, 4105, 8211, 8300), "j92": (1, 7, 33, 8200, 16400, 33000), "drm19": (1, 5, 700)}


def _state(torch, rc, n, Ts, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    Y = rng.dirichlet(np.full(rc.nsp, 0.4), n).T
    if n > 4:                                      # absent species, and one cell of a single species
        Y[:, :n // 4] = np.where(Y[:, :n // 4] < 0.02, 0.0, Y[:, :n // 4])
        Y[:, 0] = 0.0
        Y[0, 0] = 1.0
    Y = Y / Y.sum(axis=0)
    dev = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")
    T, p, Y = dev(rng.uniform(Ts[0], Ts[1], n)), dev(10.0 ** rng.uniform(4.0, 5.3, n)), dev(Y)
    rho, u = rc.thermo_from_pT(p, T, Y)
    if n > 6:
        rho[5] = -1.0                              # an invalid density keeps its input
    dt_chem = dev(np.where(rng.uniform(size=n) < 0.7, -1.0, 10.0 ** rng.uniform(-9.0, -6.5, n)))
    return rho, u, T, p, Y, dt_chem


def _run(torch, rc, state, dt):
    rho, u = state[:2]
    T, p, Y, dtc = (t.clone() for t in state[2:])
    st = torch.full((T.shape[0],), -7, dtype=torch.int32, device="cuda")
    cnt = torch.zeros((6, T.shape[0]), dtype=torch.int32, device="cuda")
    rc.update(rho, u, T, p, Y, dtc, dt, status=st, T_frozen=450.0, cell_counters=cnt)
    torch.cuda.synchronize()
    return dict(T=T, p=p, massf=Y, dt_chem=dtc, status=st, counters=cnt)


@pytest.mark.parametrize("name,n", [(m, n) for m in sorted(MECHS) for n in SIZES.get(m, (1, 260))])
def test_lanes_per_cell_change_no_result(name, n):
    import torch
    from gdtk_gb300 import lib
    from gdtk_gb300.cells import ReactorCells
    Tlo, Thi, dt = MECHS[name]
    rc = ReactorCells(mech(name + "-gas.lua"), mech(name + "-chem.lua"))
    state = _state(torch, rc, n, (Tlo, Thi), seed=n)
    got = _run(torch, rc, state, dt)
    assert lib().chem_reactor_configure(rc.reactor.id, 64, 1) == 0
    ref = _run(torch, rc, state, dt)
    assert lib().chem_reactor_configure(rc.reactor.id, 0, 0) == 0
    for k in ref:
        assert torch.equal(got[k], ref[k]), k
    if n > 6:
        assert int(ref["status"][5]) == 5
