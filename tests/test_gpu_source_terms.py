"""Species source terms by the mechanism-specialised kernel at the edges of a launch, against the oracle's right-hand side.

One cell, one warp's and one block's cells and one more or less, more than one turn of the grid; absent species, an invalid
density (status bad_input), with and without a status array.  Rate constants are in log form: |ln k| up to about 100 with
some ulps each is 1e-13 relative, and q - L cancels, so the tolerance is 1e-11 of q + L (as the oracle gives them)."""
import numpy as np
import pytest

import oracle
from conftest import mech
from test_gpu_large_mechanism import _cells

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["park5", "j92", "drm19"])
def test_source_terms_at_launch_edges(name):
    import torch
    from gdtk_gb300.cells import ReactorCells
    rc = ReactorCells(mech(name + "-gas.lua"), mech(name + "-chem.lua"))
    orc = oracle.Oracle(mech(name + "-gas.lua"), mech(name + "-chem.lua"))
    n = 60001
    T, p, Y = _cells(name, rc, n, seed=29)
    Y[0, ::7] = 0.0
    Y = np.ascontiguousarray(Y / Y.sum(axis=0))
    dev = lambda a: torch.tensor(a, dtype=torch.float64, device="cuda")
    dT, dp, dY = dev(T), dev(p), dev(Y)
    rho, _ = rc.thermo_from_pT(dp, dT, dY)
    rho[3] = -1.0
    st = torch.full((n,), -7, dtype=torch.int32, device="cuda")
    full = rc.source_terms(rho, dT, dY, status=st)
    torch.cuda.synchronize()
    assert int(st[3]) == 5 and int((st == 0).sum()) == n - 1
    for lo, m in ((0, 1), (4, 31), (4, 33), (9, 255), (9, 257), (1000, 40001)):
        part = rc.source_terms(rho[lo:lo + m].contiguous(), dT[lo:lo + m].contiguous(), dY[:, lo:lo + m].contiguous())
        assert torch.equal(part, full[:, lo:lo + m]), (lo, m)
    full, rho_h = full.cpu().numpy(), rho.cpu().numpy()
    M = np.asarray(orc.M)
    for i in list(range(0, 3)) + list(range(4, 60)) + list(range(1000, n, 997)):
        c = rho_h[i] * Y[:, i] / M
        c[c < 1e-30] = 0.0
        q, L, _, _ = orc.split_rates(T[i], c)
        assert (np.abs(full[:, i] - (q - L) * M) <= 1e-11 * (q + L) * M + 1e-30).all(), i
