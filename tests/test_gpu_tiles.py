"""The pressure solver on 2x2x2 tiles (the default; odd dimensions leave pads) against the same solver in the cell hyperplane order (forced by a sweep
variant): the same bits on every shape, at the edges of the tile hyperplanes, with
few and many grids, walls on graded grids and a hierarchy."""
import numpy as np
import pytest

from mglet_gb300 import abi, cases
from test_oracle_levels import prepare_levels

pytestmark = pytest.mark.gpu


def _run(gpu_lib, case, plane_order, nouter=3):
    prm = abi.make_flow_params(gmol=1e-3, epcorr=1e-10, nouter=nouter, ninner=3, form=abi.FORM_MIXED)
    g = gpu_lib.Solver(case, prm)
    if plane_order:
        g.force_variant("mx_sip_sweep", 0)
    u, v, w, p = cases.taylor_green(case)
    u, v, w = cases.add_noise(case, (u, v, w), amplitude=1e-2, seed=5)
    for nm, a in zip("UVWP", (u, v, w, p)):
        g.set(nm, a)
    if case.iparent is not None:
        g.set_hierarchy(case.iparent, case.position)
        for lvl in (1, 2):
            g.connect(lvl, 2, v1="U", v2="V", v3="W", s1="P", corners=True)
        prepare_levels(g, case)
    else:
        g.connect(0, 2, "U", "V", "W", "P", corners=True)
    rk = gpu_lib.rk_scheme("williamson")
    st = [g.timeintegrate_flow(1, 1, 0.0, 5e-4, irk, rk) for irk in (1, 2, 3)]
    out = [g.get(nm) for nm in ("U", "V", "W", "P", "DP")]
    g.close()
    return [(s.nouter_done, s.maxrhs) for s in st], out


def _same(gpu_lib, case):
    (sa, a), (sb, b) = _run(gpu_lib, case, False), _run(gpu_lib, case, True)
    assert sa == sb
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


# the smallest tile grid, one tile wide in each direction, hyperplanes of one to
# three warps, shapes beyond the packed cell tables, two sets of warps and one
@pytest.mark.parametrize("tiles,shape", [
    ((2, 1, 1), (2, 2, 2)), ((1, 2, 2), (2, 16, 6)), ((2, 1, 2), (12, 2, 8)), ((2, 2, 1), (6, 10, 2)),
    ((2, 2, 2), (24, 24, 24)), ((1, 2, 1), (32, 28, 36)), ((7, 7, 7), (8, 10, 12)),
    ((8, 7, 6), (20, 24, 16)),
    # pads on one axis, two and all; last tiles that are also first ones
    ((2, 2, 1), (3, 2, 2)), ((1, 2, 2), (2, 5, 4)), ((2, 1, 2), (4, 2, 7)), ((2, 2, 2), (21, 26, 19)),
    ((1, 1, 1), (3, 3, 3)), ((2, 1, 1), (33, 31, 35)), ((7, 7, 7), (9, 8, 11)), ((3, 2, 3), (5, 25, 13))])
def test_tiles_match_the_cell_order(gpu_lib, tiles, shape):
    ni, nj, nk = shape
    _same(gpu_lib, cases.periodic_box(*tiles, n=ni, nj=nj, nk=nk))


@pytest.mark.parametrize("shape", [(10, 10, 10), (9, 10, 11), (7, 9, 5)])
def test_tiles_match_with_walls_on_graded_grids(gpu_lib, shape):
    walls = {1: abi.BC_FIX, 2: abi.BC_OP1, 3: abi.BC_NOS, 4: abi.BC_SLI}
    ni, nj, nk = shape
    box = cases.periodic_box(3, 2, 2, n=ni, nj=nj, nk=nk, length=(2.0, 2.0, 1.0), walls=walls)
    _same(gpu_lib, cases.stretch(box))


@pytest.mark.parametrize("scale", [1.0, 1e-22, 1e-36, 1e-43, 1e-300, 1e30])
def test_divergence_split_over_the_range(gpu_lib, scale):
    """The divergence split into two floats by integer arithmetic against the cell
    order's casts, where the second float is normal, subnormal or lost and where the
    values leave the floats' range."""
    case = cases.periodic_box(2, 1, 1, n=6)
    out = []
    for plane in (False, True):
        g = gpu_lib.Solver(case, abi.make_flow_params(gmol=1e-3, epcorr=1e-10, nouter=1, ninner=1,
                                                      form=abi.FORM_MIXED))
        if plane:
            g.force_variant("mx_order", 0)
        rng = np.random.default_rng(2)
        for nm in "UVW":
            a = scale * rng.standard_normal(case.idim3d)
            a[rng.random(a.size) < 0.3] = 0.0
            g.set(nm, a)
        g.timeintegrate_flow(1, 1, 0.0, 5e-4, 1, gpu_lib.rk_scheme("williamson"))
        out.append([g.get(nm) for nm in ("U", "V", "W", "P", "DP")])
        g.close()
    for x, y in zip(*out):
        assert np.array_equal(x, y, equal_nan=True)


def test_tiles_match_on_a_hierarchy(gpu_lib):
    _same(gpu_lib, cases.refined_box(2, 2, 2, n=8, refine=(1,)))
