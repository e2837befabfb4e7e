"""No cell's result may depend on how many lanes integrate it.

The library spreads a cell over 4, 8, 16 or 32 lanes, or gives it one thread, from the batch's size.  A batch large
enough for the fewest lanes is compared, bit for bit, with its own slices of sizes that take every other choice
(among them one warp's cells and one more or less), and the Runge-Kutta mechanisms also with the
one-thread-per-cell kernel, which chem_reactor_configure with a block size asks for.  The cells include absent
species, a single species, an invalid density, frozen cells and carried step sizes; a batch's last cells
are regrouped over more lanes while it runs.
"""
import numpy as np
import pytest

from conftest import mech

pytestmark = pytest.mark.gpu

# mechanism: T range, interval, batch, slices.  RKF (backward rates from K_c and given), alpha-QSS with tight
# coupling, falloff rates, forward rates in other forms
MECHS = {"park5": (2000.0, 8000.0, 2.0e-7, 24000, (1, 3, 33, 700, 2050, 5000, 9000)),
         "gupta5": (2000.0, 6000.0, 1.0e-7, 24000, (1, 1100, 5100)),
         "n2": (3000.0, 6000.0, 1.0e-6, 24000, (2, 1100, 5100)),
         "j92": (400.0, 2600.0, 2.0e-7, 72000, (1, 7, 33, 700, 9001, 45001)),
         "stanford": (1000.0, 2400.0, 1.0e-7, 72000, (5, 2000, 20001, 45001)),
         "drm19": (1000.0, 2400.0, 1.0e-7, 45000, (1, 9, 700, 6001, 15001)),
         "h2o2forms": (900.0, 2400.0, 1.0e-7, 400, (1, 33))}


def _state(torch, rc, n, Ts, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    Y = rng.dirichlet(np.full(rc.nsp, 0.4), n).T
    Y[:, :n // 4] = np.where(Y[:, :n // 4] < 0.02, 0.0, Y[:, :n // 4])   # absent species
    Y[:, 3] = 0.0                                                        # a single species
    Y[0, 3] = 1.0
    Y = Y / Y.sum(axis=0)
    dev = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")
    T, p, Y = dev(rng.uniform(Ts[0], Ts[1], n)), dev(10.0 ** rng.uniform(4.0, 5.3, n)), dev(Y)
    rho, u = rc.thermo_from_pT(p, T, Y)
    rho[5] = -1.0
    dt_chem = dev(np.where(rng.uniform(size=n) < 0.7, -1.0, 10.0 ** rng.uniform(-9.0, -6.5, n)))
    return rho, u, T, p, Y, dt_chem


def _run(torch, rc, state, dt, lo=0, n=None):
    n = state[0].shape[0] if n is None else n
    rho, u, T, p, Y, dtc = (t[..., lo:lo + n].contiguous().clone() for t in state)
    st = torch.full((n,), -7, dtype=torch.int32, device="cuda")
    cnt = torch.zeros((6, n), dtype=torch.int32, device="cuda")
    rc.update(rho, u, T, p, Y, dtc, dt, status=st, T_frozen=450.0, cell_counters=cnt)
    torch.cuda.synchronize()
    return dict(T=T, p=p, massf=Y, dt_chem=dtc, status=st, counters=cnt)


@pytest.mark.parametrize("name", sorted(MECHS))
def test_lanes_per_cell_change_no_result(name):
    import torch
    from gdtk_gb300 import lib
    from gdtk_gb300.cells import ReactorCells
    Tlo, Thi, dt, n, slices = MECHS[name]
    rc = ReactorCells(mech(name + "-gas.lua"), mech(name + "-chem.lua"))
    state = _state(torch, rc, n, (Tlo, Thi), seed=n)
    ref = _run(torch, rc, state, dt)
    assert int(ref["status"][5]) == 5 and int((ref["status"] == 0).sum()) > 0.9 * n * (0.95 if name == "j92" else 1.0)
    for k, m in enumerate(slices):
        lo = min(3 + 40 * k, n - m)
        got = _run(torch, rc, state, dt, lo, m)
        for key in ref:
            assert torch.equal(got[key], ref[key][..., lo:lo + m]), (m, key)
    if rc.method == "rkf":
        assert lib().chem_reactor_configure(rc.reactor.id, 64, 1) == 0
        got = _run(torch, rc, state, dt, 0, 5000)
        assert lib().chem_reactor_configure(rc.reactor.id, 0, 0) == 0
        for key in ref:
            assert torch.equal(got[key], ref[key][..., :5000]), key
