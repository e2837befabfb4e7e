"""One, two or four warps per cell (chem_kernels.cu's chem_warp_kernel): the number, which follows from the batch and from
shared memory, changes no result; and factors that fill a table row, with coefficients that are no power of two, and one
too large for it.

Slices of one cell up to a few cells per SM take four warps a cell, whole batches two (the acetylene mechanism) or one
(small mechanisms with GDTK_CHEM_WARP_PER_CELL, a slice of which takes two), longest first; every output is compared bit for bit, among them an invalid density
and frozen cells."""
import numpy as np
import pytest

from conftest import mech
from test_gpu_large_mechanism import WARP_PER_CELL, _cells, pair
from test_gpu_parity import assert_parity, run_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,n,flags,dt", [("c2h2", 3100, 3, 1.0e-7), ("park5", 6200, 3 | WARP_PER_CELL, 1.0e-6),
                                             ("j92", 6200, 3 | WARP_PER_CELL, 1.0e-7)])
def test_number_of_warps_changes_no_result(name, n, flags, dt):
    import torch
    from gdtk_gb300.cells import ReactorCells
    from gdtk_gb300.workloads import acetylene_cells
    rc = ReactorCells(mech(name + "-gas.lua"), mech(name + "-chem.lua"))
    T, p, Y = (acetylene_cells(rc.species_names, rc.mol_masses, n, seed=3) if name == "c2h2"
               else _cells(name, rc, n, seed=3))
    dev = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")
    T, p, Y = dev(T), dev(p), dev(Y)
    rho, u = rc.thermo_from_pT(p, T, Y)
    rho[2] = -1.0
    T_frozen = float(T.min()) * 1.01
    warps = set()

    def run(lo, m):
        cut = lambda t: t[..., lo:lo + m].contiguous().clone()
        a = dict(T=cut(T), p=cut(p), massf=cut(Y), dt_chem=torch.full((m,), -1.0, dtype=torch.float64, device="cuda"))
        st = torch.full((m,), -7, dtype=torch.int32, device="cuda")
        cnt = torch.zeros((6, m), dtype=torch.int32, device="cuda")
        rc.update(cut(rho), cut(u), a["T"], a["p"], a["massf"], a["dt_chem"], dt, status=st, T_frozen=T_frozen, flags=flags,
                  cell_counters=cnt)
        torch.cuda.synchronize()
        warps.add(rc.last_launch()["block"] // 32)
        return dict(a, status=st, counters=cnt)

    ref = run(0, n)
    assert int(ref["status"][2]) == 5 and int((ref["status"] == 6).sum()) >= 1
    assert int((ref["status"] == 0).sum()) > 0.9 * n
    for lo, m in ((0, 1), (1, 3), (0, 153), (7, 608), (2, 1217), (1, 4000)):
        m = min(m, n - lo)
        got = run(lo, m)
        for k in ref:
            assert torch.equal(got[k], ref[k][..., lo:lo + m]), (lo, m, k)
    assert 4 in warps and max(warps) == 16   # one cell of four warps; a full block


@pytest.mark.parametrize("ode", ["method='rkf', errTol=1.000000e-03", "method='alpha-qss', eps1=1.0e-3, eps2=5.0e-4, delta=1.0e-10, maxIters=10"])
def test_reactions_of_many_factors(tmp_path, ode):
    import oracle
    from gdtk_gb300.cells import ReactorCells
    from gdtk_gb300.workloads import air5_cells
    text = open(mech("park5-chem.lua")).read()
    assert "method='rkf', errTol=1.000000e-03" in text
    text = text.replace("method='rkf', errTol=1.000000e-03", ode)
    for k, (A, ri, rco, pi, pco) in enumerate([(1e10, "0, 1, 3, 4,", "1, 1, 1, 1,", "2, 3, 4,", "2, 1, 1,"),
                                               (1e10, "3, 4, 1,", "3, 1, 1,", "0, 2, 4,", "1, 1, 2,"),
                                               (1e-3, "2, 4,", "1, 300,", "3, 4,", "1, 301,")]):
        text += """
reaction[%d] = {
  equation = "r%d",
  type = "elementary",
  frc = {model='Arrhenius', A=%.12e, n=0.000000, C=1.000000000000e+04, rctIndex=-1},
  brc = {model='Arrhenius', A=%.12e, n=0.000000, C=1.000000000000e+04, rctIndex=-1},
  ec = {},
  reacIdx = { %s},
  reacCoeffs = { %s},
  prodIdx = { %s},
  prodCoeffs = { %s},
  label = "r%d",
}
""" % (6 + k, 6 + k, A, 0.5 * A, ri, rco, pi, pco, 6 + k)
    chem = str(tmp_path / "chem.lua")
    open(chem, "w").write(text)
    rc, orc = ReactorCells(mech("park5-gas.lua"), chem), oracle.Oracle(mech("park5-gas.lua"), chem)
    T, p, Y = air5_cells(384, seed=9)
    thin = p / (8.314 * T) < 0.9   # the 300th power of a concentration above 1 mol/m^3 overflows: rubbish in any kernel
    T, p, Y = T[thin], p[thin], np.ascontiguousarray(Y[:, thin])
    g, o, _, _ = run_pair(rc, orc, T, p, Y, 1.0e-7, flags=3 | WARP_PER_CELL)
    assert_parity(g, o)
    assert (g["status"] == 0).mean() > 0.95
