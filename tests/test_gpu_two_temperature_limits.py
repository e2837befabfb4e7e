"""The two-temperature update at input states whose relaxation times have no value: T of zero or below gives a time that is no
number, which relaxes nothing, and the cell is updated; an infinite pressure gives what a very large one does, as its
Millikan-White times are both nothing beside Park's."""
import numpy as np
import pytest

from conftest import mech

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["park2t", "park2tmt"])
def test_states_without_relaxation_times(name):
    import torch
    from gdtk_gb300.cells import ReactorCells2T
    from gdtk_gb300.workloads import air2t_cells
    rc = ReactorCells2T(mech("park2t-gas.lua"), mech(name + "-chem.lua"), mech(name + "-eem.lua"))
    T, Tve, p, Y = air2t_cells(1, seed=7)
    n = 6
    dev = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")
    T, Tve, p, Y = dev(np.repeat(T, n)), dev(np.repeat(Tve, n)), dev(np.repeat(p, n)), dev(np.repeat(Y, n, axis=1))
    rho, _, _ = rc.thermo_from_pT(p, T, Tve, Y)
    if name == "park2t":
        T[1], T[2] = 0.0, -100.0
    p[3], p[4] = float("inf"), 1.0e300
    a = [T.clone(), Tve.clone(), p.clone(), Y.clone(), torch.full_like(T, -1.0)]
    st = torch.full((n,), -7, dtype=torch.int32, device="cuda")
    rc.update(rho, *a, 1.0e-7, status=st)
    torch.cuda.synchronize()
    assert bool((st == 0).all()), st
    for t in a:
        assert bool(torch.isfinite(t).all())
        assert torch.equal(t[..., 3], t[..., 4]) and torch.equal(t[..., 0], t[..., 5])
