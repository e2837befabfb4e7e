"""Pressure-dependent rates of cells with negative mass fractions, as a transport scheme's undershoots leave them: their third
bodies are those of the mass fractions as given (rate_constant.d:114-121), while the right-hand side sees the
concentrations clipped (gas_model.d:237-256).

Methane-air (Troe rates): source terms of a batch against the per-state entry point, which runs the reference-order kernel,
to 1e-9 of the cell's largest; batch and per-state updates, and the one-thread-per-cell kernel, against the oracle."""
import numpy as np
import pytest

import oracle
from conftest import mech
from test_gpu_large_mechanism import _cells
from test_gpu_parity import assert_parity, run_pair, to_dev, torch_cuda

pytestmark = pytest.mark.gpu


def test_negative_mass_fractions():
    from gdtk_gb300 import lib
    from gdtk_gb300.cells import ReactorCells
    from gdtk_gb300.gas import GasModel, GasState, ThermochemicalReactor
    torch = torch_cuda()
    gas, chem = mech("drm19-gas.lua"), mech("drm19-chem.lua")
    rc, orc = ReactorCells(gas, chem), oracle.Oracle(gas, chem)
    n = 24
    T, p, Y = _cells("drm19", rc, n, seed=47)
    rng = np.random.Generator(np.random.PCG64(5))
    minor = [i for i in range(rc.nsp) if Y[i].max() < 0.01]
    for k in range(n):   # two minor species negative, the largest makes up for it
        for i in rng.choice(minor, 2, replace=False):
            Y[i, k] = -10.0 ** rng.uniform(-4.0, -3.4)   # 1e-3 together would be refused as a mass-fraction error
    Y = np.ascontiguousarray(Y / Y.sum(axis=0))
    g, o, rho, u = run_pair(rc, orc, T, p, Y, 1.0e-7)
    assert_parity(g, o)
    assert (g["status"] == 0).all()
    gm = GasModel(gas)
    reactor = ThermochemicalReactor(gm, chem)
    dT, dp, dY = to_dev(torch, T, p, Y)
    drho, _ = rc.thermo_from_pT(dp, dT, dY)
    batch = rc.source_terms(drho, dT, dY).cpu().numpy()
    for k in range(n):
        gs = GasState(gm)
        gs.p, gs.T, gs.massf = float(p[k]), float(T[k]), [float(y) for y in Y[:, k]]
        gs.update_thermo_from_pT()
        one = np.array(reactor.source_terms(gs))
        assert np.abs(batch[:, k] - one).max() <= 1e-9 * np.abs(one).max(), k
        reactor.update_state(gs, 1.0e-7)
        gs.update_thermo_from_rhou()
        assert np.abs(np.array(gs.massf) - o["massf"][k]).max() <= 1e-8 and abs(gs.T - o["T"][k]) <= 1e-7 * o["T"][k], k
    assert lib().chem_reactor_configure(rc.reactor.id, 64, 1) == 0
    assert_parity(run_pair(rc, orc, T, p, Y, 1.0e-7)[0], o)
