"""q and L sums whose terms or whose value lie at the ends of the range: the fixed-point sums of the alpha-QSS kernels
(chem_group.cuh's grp_gather, chem_kernels.cu's w_gather) leave them to the FP64 chain, so both kernels end such cells
with the status of the one-thread-per-cell kernel, whose sums are such chains.  (The reference-order kernel forms the
step otherwise, so that an infinite loss rate makes other NaNs there; a rate of -inf ends all alike.)

Air with reactions added: one whose forward rate constant overflows to -inf, of species with coefficients of 2 (their
scaling must not carry the sign out of the word); and eight first-order ones whose rates are finite and whose sum is not."""
import numpy as np
import pytest

from conftest import mech
from test_gpu_long_sums import QSS, _copies, _pair
from test_gpu_parity import run_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what", ["-inf", "sum"])
def test_statuses_at_the_ends_of_the_range(tmp_path, what):
    from gdtk_gb300 import lib
    from gdtk_gb300.workloads import air5_cells
    text = open(mech("park5-chem.lua")).read()
    assert "method='rkf', errTol=1.000000e-03" in text
    text = text.replace("method='rkf', errTol=1.000000e-03", QSS)
    if what == "-inf":   # 2 NO <=> 2 O2, kf = -1e300 T^4
        text = _copies(text, 6, 1, -1.0e300, 4.0, 0.0, [(2, 2)], [(1, 2)])
    else:                # N2 <=> NO, kf = 1e307
        text = _copies(text, 6, 8, 1.0e307, 0.0, 0.0, [(0, 1)], [(2, 1)])
    rc, orc = _pair(tmp_path, "park5", text)
    T, p, Y = air5_cells(128, seed=4)
    if what == "sum":
        p = np.full_like(p, 4.0e5)
    ref = run_pair(rc, orc, T, p, Y, 1.0e-7, kernel="reference_order")[0]["status"]
    got = {"group": run_pair(rc, orc, T, p, Y, 1.0e-7)[0]["status"], "warps": run_pair(rc, orc, T, p, Y, 1.0e-7, flags=3 | 16)[0]["status"]}
    assert lib().chem_reactor_configure(rc.reactor.id, 64, 1) == 0
    want = run_pair(rc, orc, T, p, Y, 1.0e-7)[0]["status"]
    assert (want != 0).all() and (what == "sum" or np.array_equal(want, ref))
    for k, g in got.items():
        assert np.array_equal(g, want), (k, g, want)
