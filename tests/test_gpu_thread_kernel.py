"""The one-thread-per-cell kernel of the alpha-QSS mechanisms, which an explicit launch shape, lane statistics and the autotuner
reach (every size of batch takes the group kernel by default): parity with the oracle, and the refill chunk, which
that kernel alone has, changing no result."""
import numpy as np
import pytest

from conftest import mech
from test_gpu_large_mechanism import _cells, pair
from test_gpu_parity import assert_parity, run_pair, to_dev, torch_cuda

pytestmark = pytest.mark.gpu


@pytest.fixture
def shaped():
    """pair(name) with the launch shape (64, 1), the default shape and refill afterwards."""
    from gdtk_gb300 import lib
    made = []

    def make(name):
        rc, orc = pair(name)
        assert lib().chem_reactor_configure(rc.reactor.id, 64, 1) == 0
        made.append(rc)
        return rc, orc
    yield make
    for rc in made:
        assert lib().chem_reactor_set_refill_chunk(rc.reactor.id, 0) == 0
        assert lib().chem_reactor_configure(rc.reactor.id, 0, 0) == 0


@pytest.mark.parametrize("name,dt", [("j92", 1.0e-6), ("drm19", 1.0e-7), ("h2o2forms", 1.0e-7)])
def test_parity_with_the_oracle(shaped, name, dt):
    rc, orc = shaped(name)
    if name == "h2o2forms":
        rng = np.random.Generator(np.random.PCG64(3))
        n = 256
        T, p = rng.uniform(1000.0, 2400.0, n), 10.0 ** rng.uniform(4.0, 5.3, n)
        Y = np.ascontiguousarray(rng.dirichlet(np.full(rc.nsp, 0.4), n).T)
    else:
        T, p, Y = _cells(name, rc, 256, seed=19)
    g, o, _, _ = run_pair(rc, orc, T, p, Y, dt)
    assert_parity(g, o)
    assert rc.last_launch()["block"] <= 64


@pytest.mark.parametrize("chunk", [32, 128, 4096])
def test_refill_chunk_changes_no_result(shaped, chunk):
    from gdtk_gb300 import lib
    torch = torch_cuda()
    rc, _ = shaped("j92")
    n = 30000   # more than one turn of the resident threads
    T, p, Y = _cells("j92", rc, n, seed=72)
    dT, dp, dY = to_dev(torch, T, p, Y)
    rho, u = rc.thermo_from_pT(dp, dT, dY)
    outs = []
    for cells in (0, chunk):
        assert lib().chem_reactor_set_refill_chunk(rc.reactor.id, cells) == 0
        a = [dT.clone(), dp.clone(), dY.clone(), torch.full((n,), -1.0, dtype=torch.float64, device="cuda")]
        st = torch.full((n,), -7, dtype=torch.int32, device="cuda")
        rc.update(rho, u, *a, 1.0e-7, status=st)
        torch.cuda.synchronize()
        outs.append(a + [st])
    last = rc.last_launch()
    assert last["grid"] * last["block"] < n and int((outs[0][-1] == 0).sum()) > 0.95 * n
    for a, b in zip(*outs):
        assert torch.equal(a, b)


def test_autotuner_times_no_refill_chunk_of_the_librarys_choice(tmp_path, monkeypatch):
    from gdtk_gb300 import autotune
    torch = torch_cuda()
    monkeypatch.setenv("GDTK_JIT_CACHE", str(tmp_path))
    monkeypatch.setattr(autotune, "SHAPES", [(0, 0)])
    rc, _ = pair("park5")
    T, p, Y = _cells("park5", rc, 512, seed=7)
    dT, dp, dY = to_dev(torch, T, p, Y)
    rho, u = rc.thermo_from_pT(dp, dT, dY)
    sample = dict(rho=rho, u=u, T=dT, p=dp, massf=dY, dt_chem=torch.full((512,), -1.0, dtype=torch.float64, device="cuda"))
    _, _, results = autotune.tune(rc, sample, 1.0e-7, tag="test", allow_warp=False)
    assert [(r["order"], r["refill_chunk"]) for r in results] == [(name, 0) for name in autotune.ORDERS]
