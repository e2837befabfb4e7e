"""Surrogate predictions written over the features they are made from (chem_surrogate_predict's out and X may overlap).

The one-kernel network writes a tile's rows while other blocks may not have read theirs yet, so where the arrays overlap
the features are gathered first; rows of one length over themselves need not be.  The activations' BF16 roundings may differ
(2^-6 of the norm allowed, as for a few layers of 2^-8 each)."""
import ctypes

import numpy as np
import pytest

from conftest import mech

pytestmark = pytest.mark.gpu

GAS = ("H2", "O2", "H2O", "OH", "O", "H")   # 9 features, padded to 16, and 7 outputs, padded to 8
CHEM = """species = {%s}
config = {
  tempLimits = {lower=300.000000, upper=50000.000000},
  odeStep = {method='alpha-qss', eps1= 1.000000e-03, eps2= 5.000000e-04, delta= 1.000000e-10, maxIters=10},
  tightTempCoupling = true,
  maxSubcycles = 10000,
  maxAttempts = 4
}
reaction = {}
reaction[1] = {
  type = "elementary",
  frc = {model='Arrhenius', A=1.0e5, n=1.0, C=1.0e3, rctIndex=-1},
  brc = {model='fromEqConst', rctIndex=-1},
  reacIdx = { 3, 0,},
  reacCoeffs = { 1, 1,},
  prodIdx = { 2, 5,},
  prodCoeffs = { 1, 1,},
}
"""


def _six_species(tmp_path):
    from gdtk_gb300.cells import ReactorCells
    gas = open(mech("stanford-gas.lua")).read()
    at = gas.index("species = {")
    gas = gas[:at] + "species = {%s}" % ", ".join("'%s'" % s for s in GAS) + gas[gas.index("}", at) + 1:]
    for name, text in (("gas", gas), ("chem", CHEM % ", ".join("[%d]='%s'" % x for x in enumerate(GAS)))):
        with open(str(tmp_path / (name + ".lua")), "w") as f:
            f.write(text)
    return ReactorCells(str(tmp_path / "gas.lua"), str(tmp_path / "chem.lua"))


@pytest.mark.parametrize("n", [1, 129, 3 * 152 * 128 + 7])
@pytest.mark.parametrize("which", ["six", "j92"])
def test_rows_over_their_features(tmp_path, which, n):
    import torch
    from gdtk_gb300 import check, lib
    from gdtk_gb300.cells import ReactorCells
    from gdtk_gb300.surrogate import ChemSurrogate
    rc = _six_species(tmp_path) if which == "six" else ReactorCells(mech("j92-gas.lua"), mech("j92-chem.lua"))
    sg = ChemSurrogate(rc, width=64, depth=2)
    nin, nout = sg.nin_pad, sg.nout_pad
    assert (nin, nout) == ((16, 8) if which == "six" else (16, 16))
    X = torch.randn(n, nin, device="cuda")
    ref = sg.predict(X)
    for shift in (0, 4 * nout, n * (nin - nout), n * nin):   # in floats from the features' start; the last only touches
        buf = torch.zeros(n * (nin + nout) + 4 * nout, device="cuda")
        buf[:n * nin] = X.ravel()
        check(lib().chem_surrogate_predict(sg.id, n, ctypes.c_void_p(buf.data_ptr()), ctypes.c_void_p(buf.data_ptr() + 4 * shift),
                                           ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "predict")
        torch.cuda.synchronize()
        out = buf[shift:shift + n * nout].view(n, nout)
        assert (out - ref).norm().item() <= 2.0 ** -6 * ref.norm().item(), shift
