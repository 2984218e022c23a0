"""Tensor copies of the flux kernel's planes need 128-byte lines: a grid whose
planes are not a whole number of lines keeps the plane loads, and its stage runs."""
import numpy as np
import pytest

from mglet_gb300 import abi, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,lines", [((10, 10, 10), False), ((8, 27, 18), False), ((2, 2, 2), False),
                                         ((8, 12, 16), True)])
def test_tensor_copies_only_of_whole_lines(gpu_lib, shape, lines):
    ni, nj, nk = shape
    case = cases.periodic_box(2, 1, 1, n=ni, nj=nj, nk=nk)
    assert ((nk + 4) * (nj + 4) * 8 % 128 == 0) == lines
    g = gpu_lib.Solver(case, abi.make_flow_params(gmol=1e-3, nouter=2, form=abi.FORM_MIXED))
    if lines:
        g.force_variant("mx_flux", 1)
    else:
        with pytest.raises(gpu_lib.MgletError):
            g.force_variant("mx_flux", 1)
    u, v, w, p = cases.taylor_green(case)
    for nm, a in zip("UVWP", (u, v, w, p)):
        g.set(nm, a)
    g.connect(0, 2, "U", "V", "W", "P", corners=True)
    g.timeintegrate_flow(1, 1, 0.0, 5e-4, 1, gpu_lib.rk_scheme("williamson"))
    assert np.all(np.isfinite(g.get("U")))
    g.close()
