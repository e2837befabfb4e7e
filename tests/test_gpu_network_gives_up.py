"""The one-kernel network when its waits give up: no output row keeps what the buffer held before, the error flag says so, and
the next launch is as any other.  And the surrogate update of such rows, which are NaN: every cell takes the FP64 update.

A launch parameter has every part of the kernel go the way of a wait that gave up, before a load or an MMA is in flight."""
import ctypes

import numpy as np
import pytest

from conftest import mech

pytestmark = pytest.mark.gpu


def _error(lib):
    err = ctypes.c_int()
    lib().gdtk_mlp_tcgen05(-1, None, ctypes.byref(err))
    return err.value


@pytest.mark.parametrize("name,width,depth", [("j92", 256, 4), ("drm19", 72, 2), ("park5", 8, 1)])
@pytest.mark.parametrize("n", [1, 130, 2 * 152 * 128 + 5])
def test_rows_become_nan(name, width, depth, n):
    import torch
    from gdtk_gb300 import check, lib
    from gdtk_gb300.cells import ReactorCells
    from gdtk_gb300.surrogate import ChemSurrogate
    sg = ChemSurrogate(ReactorCells(mech(name + "-gas.lua"), mech(name + "-chem.lua")), width=width, depth=depth)
    dims = sg.layer_dims()
    X = torch.randn(n, dims[0], device="cuda")
    ref = sg.predict(X)
    assert _error(lib) == 0
    out = torch.ones(n + 1, dims[-1], device="cuda")
    check(lib().chem_surrogate_predict_giving_up(sg.id, n, ctypes.c_void_p(X.data_ptr()), ctypes.c_void_p(out.data_ptr()),
                                                 ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "giving up")
    torch.cuda.synchronize()
    assert bool(torch.isnan(out[:n]).all()) and bool((out[n] == 1.0).all())
    assert _error(lib) != 0 and _error(lib) == 0
    assert torch.equal(sg.predict(X), ref) and _error(lib) == 0


def test_cells_of_nan_rows_take_the_fp64_update():
    import torch
    from gdtk_gb300.cells import ReactorCells
    from gdtk_gb300.surrogate import ChemSurrogate
    from gdtk_gb300.workloads import h2air_cells
    rc = ReactorCells(mech("j92-gas.lua"), mech("j92-chem.lua"))
    sg = ChemSurrogate(rc, width=64, depth=2)
    sg.set_params(np.full(sg.get_params().shape, np.nan, np.float32))
    n, dt = 500, 1.0e-7
    T, p, Y = h2air_cells(rc.species_names, rc.mol_masses, n, seed=6, gas_file=rc.gmodel.file_name)
    dev = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")
    T, p, Y = dev(T), dev(p), dev(Y)
    rho, u = rc.thermo_from_pT(p, T, Y)
    plain = [T.clone(), p.clone(), Y.clone(), torch.full_like(T, -1.0), torch.full((n,), -7, dtype=torch.int32, device="cuda")]
    gated = [t.clone() for t in plain]
    rc.update(rho, u, *plain[:4], dt, status=plain[4])
    gate = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    sg.update(rho, u, *gated[:4], dt, status=gated[4], gate=gate)
    torch.cuda.synchronize()
    assert bool((gate > 2).all())
    for a, b in zip(plain, gated):
        assert torch.equal(a, b)
