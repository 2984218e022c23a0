"""What the plain form's solve on tiles leaves in the fields a program can read, ghost
layers included, against the per-operator kernels (taken once the caller has written
a coefficient field): the same bits."""
import numpy as np
import pytest

from mglet_gb300 import abi, cases

pytestmark = pytest.mark.gpu

FIELDS = ("U", "V", "W", "P", "G", "DU", "DV", "DW", "BP", "SDIV", "UO", "VO", "WO", "DP", "HILF", "RHS",
          "RES", "GSAP", "SIPLW", "SIPLS", "SIPLB", "SIPLPR", "SIPUE", "SIPUN", "SIPUT")


def _run(gpu_lib, case, operators, kw):
    base = dict(gmol=1e-3, epcorr=1e-10, nouter=3, ninner=3, form=abi.FORM_PLAIN)
    base.update(kw)
    g = gpu_lib.Solver(case, abi.make_flow_params(**base))
    if operators:
        g.set("BP", np.ones(case.idim3d))
    for nm, a in zip("UVWP", cases.add_noise(case, cases.taylor_green(case), seed=5)):
        g.set(nm, a)
    g.connect(0, 2, "U", "V", "W", "P", corners=True)
    g.bound_flow()
    rk = gpu_lib.rk_scheme("williamson")
    done = [g.timeintegrate_flow(1, 1, 0.0, 5e-4, irk, rk).nouter_done for irk in (1, 2)]
    out = {nm: g.get(nm) for nm in FIELDS}
    g.close()
    return done, out


WALLS = {1: abi.BC_FIX, 2: abi.BC_OP1, 3: abi.BC_NOS, 4: abi.BC_SLI}


# single cells on clusters and on one SM, pairs; one exchange only; an early stop
@pytest.mark.parametrize("tiles,shape,walls,kw", [
    ((2, 1, 2), (8, 7, 6), None, {}), ((2, 1, 2), (8, 7, 6), None, dict(ninner=1)),
    ((1, 1, 1), (5, 6, 7), None, dict(ninner=2, nouter=1)), ((3, 2, 2), (10, 9, 8), WALLS, {}),
    ((3, 2, 2), (10, 9, 8), WALLS, dict(nouter=30, epcorr=1e-1)), ((5, 5, 4), (6, 5, 8), WALLS, dict(ninner=4)),
    ((7, 7, 7), (4, 5, 6), WALLS, {}), ((7, 7, 7), (4, 5, 6), None, dict(nouter=30, epcorr=1e-1))])
def test_every_field_matches_the_operators(gpu_lib, tiles, shape, walls, kw):
    ni, nj, nk = shape
    case = cases.periodic_box(*tiles, n=ni, nj=nj, nk=nk, **({"walls": walls} if walls else {}))
    if walls:
        case = cases.stretch(case)
    (da, a), (db, b) = (_run(gpu_lib, case, ops, kw) for ops in (False, True))
    assert da == db
    if "epcorr" in kw:
        assert max(da) < kw["nouter"]
    for nm in FIELDS:
        assert np.array_equal(a[nm], b[nm]), nm
