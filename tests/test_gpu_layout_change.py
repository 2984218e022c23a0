"""The mixed form's solver arrays change their layout when a plane-order variant is
forced or given back: nothing that the other layout left behind reaches a result."""
import numpy as np
import pytest

from mglet_gb300 import abi, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", ["mx_sip_sweep", "mx_order", None])
def test_pads_are_clear_after_a_run_that_went_to_nan(gpu_lib, kernel):
    """Odd dimensions leave pads in the last tiles; a run in the cell order fills the
    whole arrays, one on tiles the pads' neighbours."""
    case = cases.periodic_box(2, 1, 1, n=9, nj=8, nk=11)
    prm = abi.make_flow_params(gmol=1e-3, epcorr=1e-10, nouter=3, ninner=3, form=abi.FORM_MIXED)
    rk = gpu_lib.rk_scheme("williamson")
    fields = cases.taylor_green(case)

    def load(g):
        for nm, a in zip("UVWP", fields):
            g.set(nm, a)
        for nm in ("DU", "DV", "DW"):
            g.set(nm, case.zeros())
        g.connect(0, 2, "U", "V", "W", "P", corners=True)

    def stage(g):
        g.timeintegrate_flow(1, 1, 0.0, 5e-4, 1, rk)
        return [g.get(nm) for nm in ("U", "V", "W", "P", "DP")]

    g = gpu_lib.Solver(case, prm)
    load(g)
    want = stage(g)
    if kernel:
        g.force_variant(kernel, 0)
    load(g)
    g.set("U", np.full(case.idim3d, np.nan))
    stage(g)
    if kernel:
        g.force_variant(kernel, -1)
    load(g)
    for x, y in zip(stage(g), want):
        assert np.array_equal(x, y)
    g.close()
