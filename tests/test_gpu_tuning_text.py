"""mglet_gpu_tuning names the kernels that run, on tiles and with a plane-order
variant forced."""
import pytest

from mglet_gb300 import abi, cases

pytestmark = pytest.mark.gpu


def test_tuning_names_the_solver_in_use(gpu_lib):
    case = cases.periodic_box(2, 1, 1, n=8)
    g = gpu_lib.Solver(case, abi.make_flow_params(gmol=1e-3, form=abi.FORM_MIXED))
    for kernel, v in ((None, 0), ("mx_sip_sweep", 1), ("mx_outer", 1), ("mx_sip_pre", 0)):
        if kernel:
            g.force_variant(kernel, v)
        t = g.tuning()
        for part in ("mx_sip_pre:", "sweeps:", "mx_outer:"):
            words = t.split(part)[1].split(";")[0]
            assert ("2x2x2 tiles" in words) == (kernel is None), t
        assert "uniform classes: yes" in t and "mx_sip_solve: per-phase kernels" in t
        if kernel:
            g.force_variant(kernel, -1)
    assert "2x2x2 tiles" in g.tuning()
    g.close()
