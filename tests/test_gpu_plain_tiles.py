"""The plain form's pressure solve on tiles (the default on one level) against the
per-operator kernels (taken when the caller sets a coefficient field, here BP to the
ones it holds anyway): the same bits at the edges of the tile hyperplanes, in pairs
(even k extents) and single cells, with grids on one SM and shared by 2, 4 and 8 (row
counts that do not divide), on walls and graded
grids, and when the outer loop stops early or runs past a look at its flag."""
import numpy as np
import pytest

from mglet_gb300 import abi, cases

pytestmark = pytest.mark.gpu


def _run(gpu_lib, case, form, operators, **kw):
    base = dict(gmol=1e-3, epcorr=1e-10, nouter=3, ninner=3, form=form)
    base.update(kw)
    g = gpu_lib.Solver(case, abi.make_flow_params(**base))
    if operators:
        g.set("BP", np.ones(case.idim3d))
    u, v, w, p = cases.taylor_green(case)
    u, v, w = cases.add_noise(case, (u, v, w), amplitude=1e-2, seed=5)
    for nm, a in zip("UVWP", (u, v, w, p)):
        g.set(nm, a)
    g.connect(0, 2, "U", "V", "W", "P", corners=True)
    g.bound_flow()
    rk = gpu_lib.rk_scheme("williamson")
    st = [g.timeintegrate_flow(1, 1, 0.0, 5e-4, irk, rk) for irk in (1, 2, 3)]
    out = [g.get(nm) for nm in "UVWP"] + [case.interior(g.get(nm)) for nm in ("DP", "RHS", "RES")]
    g.close()
    return [(s.ipc, s.nouter_done, s.maxrhs, s.prefak) for s in st], out


def _same(gpu_lib, case, form, **kw):
    (sa, a), (sb, b) = (_run(gpu_lib, case, form, ops, **kw) for ops in (False, True))
    assert sa == sb
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


SHAPES = [
    ((2, 1, 1), (2, 2, 2)), ((1, 1, 1), (2, 3, 5)), ((1, 2, 2), (2, 16, 6)), ((2, 1, 2), (11, 2, 7)),
    ((2, 2, 2), (24, 24, 24)), ((1, 1, 2), (33, 29, 31)), ((1, 1, 1), (40, 36, 44)),
    ((3, 3, 3), (10, 9, 8)), ((4, 4, 4), (5, 6, 8)), ((6, 6, 5), (8, 10, 12)), ((7, 7, 7), (6, 5, 8)), ((7, 7, 7), (5, 6, 7)), ((6, 6, 5), (9, 8, 7))]


@pytest.mark.parametrize("tiles,shape", SHAPES)
def test_tiles_match_the_operators(gpu_lib, tiles, shape):
    ni, nj, nk = shape
    _same(gpu_lib, cases.periodic_box(*tiles, n=ni, nj=nj, nk=nk), abi.FORM_PLAIN)


@pytest.mark.parametrize("tiles,shape", SHAPES)
def test_contracted_tiles_within_the_bound_of_the_form(gpu_lib, tiles, shape):
    """Contraction rounds other sums than the operators do (the product with lpr
    rounds here): the form's relative 1e-12 holds against the uncontracted run."""
    ni, nj, nk = shape
    case = cases.periodic_box(*tiles, n=ni, nj=nj, nk=nk)
    (sa, a), (sb, b) = (_run(gpu_lib, case, form, False) for form in (abi.FORM_PLAIN_FMA, abi.FORM_PLAIN))
    assert [s[:2] for s in sa] == [s[:2] for s in sb]
    for x, y in zip(a[:4], b[:4]):
        assert np.linalg.norm(x - y) <= 1e-12 * np.linalg.norm(y)


@pytest.mark.parametrize("kw", [dict(), dict(nouter=30, epcorr=1e-2), dict(nouter=30, nouter_min=25, epcorr=1e30),
                                dict(ninner=1, nouter=1)])
def test_tiles_match_with_walls_on_graded_grids(gpu_lib, kw):
    walls = {1: abi.BC_FIX, 2: abi.BC_OP1, 3: abi.BC_NOS, 4: abi.BC_SLI}
    case = cases.stretch(cases.periodic_box(3, 2, 2, n=10, length=(2.0, 2.0, 1.0), walls=walls))
    _same(gpu_lib, case, abi.FORM_PLAIN, **kw)
