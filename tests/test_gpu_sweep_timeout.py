"""Failure detection without a fault: the plain form's sweeps of grids that several
SMs share wait for each other's faces with a limit.  With the test switch one wait of
each sweep runs out: the solve ends there, the call returns an error, and the next one
on the same context gives the bits of a fresh one."""
import time

import numpy as np
import pytest

from mglet_gb300 import abi, cases

pytestmark = pytest.mark.gpu


def _load(g, case):
    for nm, a in zip("UVWP", cases.taylor_green(case)):
        g.set(nm, a)
    for nm in ("DU", "DV", "DW"):
        g.set(nm, case.zeros())
    g.connect(0, 2, "U", "V", "W", "P", corners=True)


# clusters of 8, 4 and 2
@pytest.mark.parametrize("tiles", [(1, 1, 1), (3, 3, 3), (4, 4, 4)])
@pytest.mark.parametrize("form", [abi.FORM_PLAIN, abi.FORM_PLAIN_FMA])
def test_a_lost_wait_ends_the_solve(gpu_lib, tiles, form):
    case = cases.periodic_box(*tiles, n=12, nj=10, nk=9)
    prm = abi.make_flow_params(gmol=1e-3, epcorr=0.0, nouter=30, ninner=3, form=form)
    rk = gpu_lib.rk_scheme("williamson")
    out = []
    for lose in (False, True):
        g = gpu_lib.Solver(case, prm)
        if lose:
            _load(g, case)
            g.test_sweep_timeout()
            t = time.perf_counter()
            with pytest.raises(gpu_lib.MgletError) as err:
                g.timeintegrate_flow(1, 1, 0.0, 5e-4, 1, rk)
            t = time.perf_counter() - t
            assert err.value.code == abi.MGLET_ERR_CUDA and "timed out" in str(err.value)
            # one wait of about 50 ms, not one in each of the 90 forward sweeps
            assert 0.02 < t < 0.5
        _load(g, case)
        st = g.timeintegrate_flow(1, 1, 0.0, 5e-4, 1, rk)
        assert st.nouter_done == 30
        out.append([g.get(nm) for nm in ("U", "V", "W", "P", "DP")])
        g.close()
    for x, y in zip(*out):
        assert np.array_equal(x, y)


def test_the_switch_needs_shared_grids(gpu_lib):
    for tiles, form in (((6, 5, 4), abi.FORM_PLAIN), ((1, 1, 1), abi.FORM_MIXED)):
        g = gpu_lib.Solver(cases.periodic_box(*tiles, n=4), abi.make_flow_params(gmol=1e-3, form=form))
        with pytest.raises(gpu_lib.MgletError) as err:
            g.test_sweep_timeout()
        assert err.value.code == abi.MGLET_ERR_UNSUPPORTED
        g.close()
