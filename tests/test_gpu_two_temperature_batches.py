"""The two-temperature update with eight lanes per cell: no cell's result depends on the batch it lies in.

A batch that takes several turns of the resident cells is compared, bit for bit, with its own slices of one cell,
one warp's cells and one more or less, and one turn; an invalid density, absent species, a species mass of a rare
collider (below its threshold) and carried step sizes are among the cells.
"""
import numpy as np
import pytest

from conftest import mech

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["park2t", "park2tmt"])
def test_batches_change_no_result(name):
    import torch
    from gdtk_gb300.cells import ReactorCells2T
    from gdtk_gb300.workloads import air2t_cells
    rc = ReactorCells2T(mech("park2t-gas.lua"), mech(name + "-chem.lua"), mech(name + "-eem.lua"))
    n, dt = 30011, 1.0e-7
    T, Tve, p, Y = air2t_cells(n, seed=23)
    Y[3, 7] = 0.0
    Y[4, 8] = 1.0e-17
    Y = Y / Y.sum(axis=0)
    dev = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")
    T, Tve, p, Y = dev(T), dev(Tve), dev(p), dev(Y)
    rho, _, _ = rc.thermo_from_pT(p, T, Tve, Y)
    rho[5] = -1.0
    rng = np.random.Generator(np.random.PCG64(2))
    dt_chem = dev(np.where(rng.uniform(size=n) < 0.7, -1.0, 10.0 ** rng.uniform(-10.0, -6.5, n)))

    def run(lo, m):
        cut = lambda t: t[..., lo:lo + m].contiguous().clone()
        a = dict(T=cut(T), Tve=cut(Tve), p=cut(p), massf=cut(Y), dt_chem=cut(dt_chem))
        st = torch.full((m,), -7, dtype=torch.int32, device="cuda")
        u, uve = torch.zeros(m, dtype=torch.float64, device="cuda"), torch.zeros(m, dtype=torch.float64, device="cuda")
        rc.update(cut(rho), a["T"], a["Tve"], a["p"], a["massf"], a["dt_chem"], dt, status=st, u=u, u_ve=uve)
        torch.cuda.synchronize()
        return dict(a, status=st, u=u, u_ve=uve)

    ref = run(0, n)
    assert int(ref["status"][5]) == 5 and bool((ref["T"][5] == T[5]).item())
    assert int((ref["status"] == 0).sum()) > 0.95 * n
    for lo, m in ((0, 1), (5, 1), (3, 3), (4, 4), (2, 5), (1, 33), (0, 1217), (100, 9728)):
        got = run(lo, m)
        for k in ref:
            assert torch.equal(got[k], ref[k][..., lo:lo + m]), (lo, m, k)
