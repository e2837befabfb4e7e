"""Two-temperature mechanisms with stoichiometric coefficients above 126, which do not fit the packed words of the reaction
table: N2 + 130 O <=> N + N + 130 O against the same rate written with O twice, 65 each (O's net coefficient is 0 in both).
The concentrations of O lie about 1 mol/m^3.  The two differ in the order of 130 products alone, 130 ulps of the rate:
1e-11 relative is allowed, and 1e-9 in mass fractions, which are of the order of 1."""
import numpy as np
import pytest

from conftest import mech

pytestmark = pytest.mark.gpu


def _reactor(tmp_path, name, oxygen):
    from gdtk_gb300.cells import ReactorCells2T
    text = open(mech("park2t-chem.lua")).read()
    idx, co = ", ".join("3" for _ in oxygen), ", ".join(str(c) for c in oxygen)
    if oxygen:
        text += """
reaction[90] = {
  type = "elementary",
  frc = {model='Arrhenius', A=2.0e4, n=0.0, C=1.0e3, rctIndex=-1},
  brc = {model='fromEqConst', rctIndex=-1},
  reacIdx = { 0, %s,},
  reacCoeffs = { 1, %s,},
  prodIdx = { 2, %s,},
  prodCoeffs = { 2, %s,},
}
""" % (idx, co, idx, co)
    path = str(tmp_path / (name + ".lua"))
    with open(path, "w") as f:
        f.write(text)
    return ReactorCells2T(mech("park2t-gas.lua"), path, mech("park2t-eem.lua"))


def test_coefficients_above_126(tmp_path):
    import torch
    n, dt = 64, 1.0e-7
    rng = np.random.Generator(np.random.PCG64(8))
    dev = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")
    T, Tve = dev(rng.uniform(5000.0, 9000.0, n)), dev(rng.uniform(3000.0, 6000.0, n))
    Y = np.zeros((5, n))
    Y[0], Y[1], Y[3], Y[4] = 0.6, 0.1, 0.25, 0.05
    Y = dev(Y)
    p = dev(np.full(n, 1.0e5))
    rho = dev(rng.uniform(0.98, 1.01, n)) * 0.0159994 / 0.25   # c_O about 1 mol/m^3
    out = []
    for name, oxygen in (("one", (130,)), ("two", (65, 65)), ("none", ())):
        rc = _reactor(tmp_path, name, oxygen)
        a = dict(T=T.clone(), Tve=Tve.clone(), p=p.clone(), massf=Y.clone(), dt_chem=torch.full_like(T, -1.0))
        st = torch.full((n,), -7, dtype=torch.int32, device="cuda")
        rc.update(rho, a["T"], a["Tve"], a["p"], a["massf"], a["dt_chem"], dt, status=st)
        torch.cuda.synchronize()
        out.append(dict(a, status=st))
    one, two, none = out
    assert torch.equal(one["status"], two["status"])   # a cell or two takes more subcycles than the limit
    assert (one["status"] == 0).double().mean().item() > 0.9 and bool((none["status"] == 0).all())
    for k in ("T", "Tve", "p"):
        assert ((one[k] - two[k]).abs() / two[k]).max().item() <= 1.0e-9, k
    assert (one["massf"] - two["massf"]).abs().max().item() <= 1.0e-9
    assert (one["massf"] - none["massf"]).abs().max().item() > 1.0e-6   # the reaction counts
