"""Troe broadening with T3 = 0 or T1 = 0, which mechanism files use to leave a term out: exp(-T / 0) is 0
(kinetics/rate_constant.d:258-287).  The batch update and the per-state update against the oracle."""
import re

import numpy as np
import pytest

import oracle
from conftest import mech
from test_gpu_large_mechanism import _cells
from test_gpu_parity import assert_parity, run_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("zero", ["T3", "T1", "both"])
def test_broadening_term_left_out(tmp_path, zero):
    from gdtk_gb300.cells import ReactorCells
    from gdtk_gb300.gas import GasModel, GasState, ThermochemicalReactor
    text = open(mech("drm19-chem.lua")).read()
    for name in ("T3", "T1") if zero == "both" else (zero,):
        text, k = re.subn(r"\b%s=[0-9.e+-]+," % name, "%s=0.0," % name, text)
        assert k >= 5
    chem = str(tmp_path / "chem.lua")
    with open(chem, "w") as f:
        f.write(text)
    gas = mech("drm19-gas.lua")
    rc, orc = ReactorCells(gas, chem), oracle.Oracle(gas, chem)
    T, p, Y = _cells("drm19", rc, 128, seed=31)
    g, o, rho, u = run_pair(rc, orc, T, p, Y, 1.0e-7)
    assert_parity(g, o)
    assert (g["status"] == 0).all()
    gm = GasModel(gas)
    gs, reactor = GasState(gm), ThermochemicalReactor(gm, chem)
    k = int(np.abs(o["massf"].T - Y).max(axis=0).argmax())   # the cell that reacts most
    gs.p, gs.T, gs.massf = float(p[k]), float(T[k]), [float(y) for y in Y[:, k]]
    gs.update_thermo_from_pT()
    reactor.update_state(gs, 1.0e-7)
    assert np.abs(np.array(gs.massf) - o["massf"][k]).max() <= 1e-8
