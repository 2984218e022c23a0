"""The plain form's solve keeps coefficients of its own; every entry point that
writes a field by its name has to be seen by it when that field is BP or a Poisson
coefficient: the same bits as uploading what the call left in the field."""
import numpy as np
import pytest

from mglet_gb300 import abi, cases

pytestmark = pytest.mark.gpu


def _solver(gpu_lib, case):
    g = gpu_lib.Solver(case, abi.make_flow_params(gmol=1e-3, epcorr=1e-10, nouter=2, ninner=2,
                                                  form=abi.FORM_PLAIN))
    for nm, a in zip("UVWP", cases.taylor_green(case)):
        g.set(nm, a)
    g.connect(0, 2, "U", "V", "W", "P", corners=True)
    rng = np.random.default_rng(1)
    for nm in ("DU", "UO", "VO"):
        g.set(nm, 1e-3 * rng.standard_normal(case.idim3d))
    return g


def _stage(gpu_lib, g):
    st = g.timeintegrate_flow(1, 1, 0.0, 5e-4, 1, gpu_lib.rk_scheme("williamson"))
    return [st.maxrhs] + [g.get(nm) for nm in "UVWP"]


@pytest.mark.parametrize("name,call", [
    ("GSAP", lambda g: g.rkstep("GSAP", "DU", "UO", 0.5, 1.0)),
    ("SIPLPR", lambda g: g.rkstep("SIPLPR", "DU", "UO", 0.5, 1.0)),
    ("GSAP", lambda g: g.rkstep("DU", "GSAP", "UO", 0.5, 1.0)),
    ("BP", lambda g: g.rkstep("BP", "DU", "UO", 0.5, 1.0)),
    ("GSAP", lambda g: g.divcal("GSAP", -100.0)),
    ("GSAP", lambda g: g.laplacephi("GSAP", "VO")),
    ("SIPLPR", lambda g: g.connect(0, 2, s1="SIPLPR")), ("GSAP", lambda g: g.connect(0, 2, s1="GSAP")),
    ("BP", lambda g: g.connect(0, 2, s1="BP", corners=True))])
def test_a_written_coefficient_is_used(gpu_lib, name, call):
    case = cases.periodic_box(2, 1, 1, n=8)
    a = _solver(gpu_lib, case)
    call(a)
    value, du = a.get(name), a.get("DU")
    b = _solver(gpu_lib, case)
    b.set(name, value)
    b.set("DU", du)
    for x, y in zip(_stage(gpu_lib, a), _stage(gpu_lib, b)):
        assert np.array_equal(x, y, equal_nan=True)
    a.close()
    b.close()


@pytest.mark.parametrize("name,kept", [("BP", True), ("GSAP", True), ("SIPLPR", False), ("P", True)])
def test_connecting_ghosts_keeps_the_solve_on_tiles(gpu_lib, name, kept):
    case = cases.periodic_box(2, 1, 1, n=8)
    n = []
    for call in (False, True):
        g = _solver(gpu_lib, case)
        if call:
            g.connect(0, 2, s1=name)
        n0 = g.launches
        _stage(gpu_lib, g)
        n.append(g.launches - n0)
        g.close()
    assert (n[0] == n[1]) == kept
