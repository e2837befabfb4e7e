"""q and L sums of many terms of one size, against the oracle.

The alpha-QSS kernels add a sum's terms in 64-bit fixed point with room for 64 of the largest one (chem_group.cuh's
grp_gather, chem_kernels.cu's w_gather); longer sums are FP64 chains.  A mechanism with many copies of one reaction has
sums of that many equal terms: 60, 62 (64 entries for one sum, 66 for another) and 100 copies, of a reaction with coefficients of 1
and of one with a 2, in the kernel with a group of lanes per cell; 990 copies of a reaction of six species in the one
for large mechanisms, whose lanes then add parts of 94 terms."""
import numpy as np
import pytest

import oracle
from conftest import mech
from test_gpu_parity import assert_parity, run_pair

pytestmark = pytest.mark.gpu

QSS = "method='alpha-qss', eps1= 1.000000e-03, eps2= 5.000000e-04, delta= 1.000000e-10, maxIters=10"


def _copies(text, first, count, A, n, C, reac, prod):
    side = lambda s: (", ".join(str(i) for i, _ in s), ", ".join(str(c) for _, c in s))
    (ri, rc), (pi, pc) = side(reac), side(prod)
    for k in range(count):
        text += """
reaction[%d] = {
  type = "elementary",
  frc = {model='Arrhenius', A=%.12e, n=%.6f, C=%.12e, rctIndex=-1},
  brc = {model='fromEqConst', rctIndex=-1},
  reacIdx = { %s,},
  reacCoeffs = { %s,},
  prodIdx = { %s,},
  prodCoeffs = { %s,},
}
""" % (first + k, A, n, C, ri, rc, pi, pc)
    return text


def _pair(tmp_path, gas, text):
    from gdtk_gb300.cells import ReactorCells
    chem = str(tmp_path / "chem.lua")
    with open(chem, "w") as f:
        f.write(text)
    return ReactorCells(mech(gas + "-gas.lua"), chem), oracle.Oracle(mech(gas + "-gas.lua"), chem)


@pytest.mark.parametrize("count", [60, 62, 100])
@pytest.mark.parametrize("coeff", [1, 2])
def test_copies_of_a_reaction(tmp_path, count, coeff):
    from gdtk_gb300.workloads import air5_cells
    text = open(mech("park5-chem.lua")).read()
    assert "method='rkf', errTol=1.000000e-03" in text
    text = text.replace("method='rkf', errTol=1.000000e-03", QSS)
    if coeff == 1:    # N2 + O <=> NO + N
        text = _copies(text, 6, count, 6.4e11, -1.0, 3.84e4, [(0, 1), (4, 1)], [(2, 1), (3, 1)])
    else:             # N2 + O2 <=> 2 NO
        text = _copies(text, 6, count, 1.0e9, 0.0, 6.0e4, [(0, 1), (1, 1)], [(2, 2)])
    rc, orc = _pair(tmp_path, "park5", text)
    T, p, Y = air5_cells(384, seed=13)
    g, o, _, _ = run_pair(rc, orc, T, p, Y, 1.0e-7)
    assert_parity(g, o)
    assert (g["status"] == 0).mean() > 0.95


def test_a_thousand_copies_in_the_large_mechanism_kernel(tmp_path):
    from gdtk_gb300.workloads import h2air_cells
    text = open(mech("j92-chem.lua")).read()
    # O + H2 + HO2 <=> H + O2 + H2O
    text = _copies(text, 900, 990, 1.0e9, 0.0, 3.0e3, [(12, 1), (2, 1), (5, 1)], [(11, 1), (1, 1), (3, 1)])
    rc, orc = _pair(tmp_path, "j92", text)
    assert rc.nr > 1000
    T, p, Y = h2air_cells(rc.species_names, rc.mol_masses, 192, seed=5, gas_file=rc.gmodel.file_name)
    g, o, _, _ = run_pair(rc, orc, T, p, Y, 1.0e-7)
    assert_parity(g, o)
    assert (g["status"] == 0).mean() > 0.95
