"""Warps per cell with GDTK_CHEM_WARP_PER_CELL: a mechanism of up to 16 reactions and species gets one, of up to 32 two, a larger
one four while the batch is small; and batches around one turn of the resident cells, whose first cells are dealt over the
SMs, give each cell what it has alone."""
import numpy as np
import pytest

from conftest import mech
from test_gpu_large_mechanism import WARP_PER_CELL
from test_gpu_parity import _premixed_cells

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,warps", [("park5", 1), ("h2o2forms", 1), ("stanford", 2), ("j92", 4), ("drm19", 4)])
def test_warps_per_cell_by_the_mechanism(name, warps):
    import torch
    from gdtk_gb300.cells import ReactorCells
    rc = ReactorCells(mech(name + "-gas.lua"), mech(name + "-chem.lua"))
    n = 152 * 16 + 70
    majors = {"park5": {"N2": 3.0, "O2": 1.0}, "drm19": {"CH4": 1.0, "O2": 2.0, "N2": 7.52}}.get(name, {"H2": 1.0, "O2": 1.0})
    T, p, Y = _premixed_cells(rc.species_names, rc.mol_masses, n, seed=2, majors=majors)
    dev = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")
    T, p, Y = dev(T), dev(p), dev(Y)
    rho, u = rc.thermo_from_pT(p, T, Y)

    def run(lo, m, flags):
        a = [t[..., lo:lo + m].contiguous().clone() for t in (T, p, Y)] + [torch.full((m,), -1.0, dtype=torch.float64, device="cuda")]
        st = torch.full((m,), -7, dtype=torch.int32, device="cuda")
        rc.update(rho[lo:lo + m].contiguous(), u[lo:lo + m].contiguous(), *a, 1.0e-8, status=st, flags=flags)
        torch.cuda.synchronize()
        return a + [st]

    ref = run(0, n, 3 | WARP_PER_CELL | 8)   # in index order
    assert int((ref[-1] == 0).sum()) > 0.95 * n
    for m in (n, 152 * 16, 152 * 16 + 1, 152, 151):
        for a, b in zip(run(0, m, 3 | WARP_PER_CELL), ref):
            assert torch.equal(a, b[..., :m]), m
    run(5, 1, 3 | WARP_PER_CELL)
    assert rc.last_launch()["block"] == 32 * warps
