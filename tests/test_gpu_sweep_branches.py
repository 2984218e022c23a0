"""Every branch of the dispatch of the solves on tiles and of the mixed fluxes, each at
a size that takes it: against the per-operator kernels (plain form), the cell
hyperplane order and the tensor copies (mixed form), the same bits."""
import numpy as np
import pytest

from mglet_gb300 import abi, cases
from test_gpu_plain_tiles import _same as plain_same
from test_gpu_tiles import _same as mixed_same
from test_oracle_gc_levels import gc_hierarchy, load_gc
from test_oracle_ghostcell import load, random_fields
from test_oracle_levels import _fine, _g3, prepare_levels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles,shape", [
    # one SM a grid, two sets of warps of up to 544 and 1024 threads; one set where two do not fit
    ((5, 5, 4), (6, 7, 8)), ((5, 5, 4), (24, 24, 24)), ((5, 4, 4), (29, 28, 27)),
    # single cells, one set of up to 320, 544 and 1024 threads
    ((6, 6, 5), (14, 15, 13)), ((6, 6, 5), (20, 20, 20)), ((6, 6, 5), (28, 28, 27)),
    # pairs, one set of up to 320, 544 and 1024 threads
    ((7, 7, 7), (18, 16, 18)), ((61, 5, 1), (32, 32, 34)), ((61, 5, 1), (27, 27, 54))])
def test_plain_sweeps_match_the_operators(gpu_lib, tiles, shape):
    ni, nj, nk = shape
    plain_same(gpu_lib, cases.periodic_box(*tiles, n=ni, nj=nj, nk=nk), abi.FORM_PLAIN)


# many grids with more than 160 threads a grid, without and with pads
@pytest.mark.parametrize("tiles,shape", [((7, 7, 7), (28, 28, 28)), ((7, 7, 7), (27, 28, 29))])
def test_mixed_sweeps_match_the_cell_order(gpu_lib, tiles, shape):
    ni, nj, nk = shape
    mixed_same(gpu_lib, cases.periodic_box(*tiles, n=ni, nj=nj, nk=nk))


def _mixed(gpu_lib, case, force, setup, nouter=3):
    g = gpu_lib.Solver(case, abi.make_flow_params(gmol=1e-2, epcorr=1e-12, nouter=nouter, ninner=3,
                                                  form=abi.FORM_MIXED))
    if force:
        g.force_variant(*force)
    setup(g)
    rk = gpu_lib.rk_scheme("williamson")
    st = [g.timeintegrate_flow(1, 1, 0.0, 2e-3, irk, rk) for irk in (1, 2, 3)]
    out = [g.get(nm) for nm in ("U", "V", "W", "P", "DP")]
    g.close()
    return [(s.nouter_done, s.maxrhs) for s in st], out


def _same(a, b):
    assert a[0] == b[0]
    for x, y in zip(a[1], b[1]):
        assert np.all(np.isfinite(x)) and np.array_equal(x, y)


# one slab of all 576 columns (many grids), slabs of few rows (few grids)
@pytest.mark.parametrize("walls", [None, {1: abi.BC_FIX, 4: abi.BC_SLI, 5: abi.BC_NOS}])
@pytest.mark.parametrize("tiles,shape", [((8, 8, 5), (4, 24, 24)), ((2, 1, 1), (8, 12, 16))])
def test_plane_loads_match_the_tensor_copies(gpu_lib, tiles, shape, walls):
    ni, nj, nk = shape
    case = cases.periodic_box(*tiles, n=ni, nj=nj, nk=nk, **({"walls": walls} if walls else {}))
    f = cases.add_noise(case, cases.taylor_green(case), amplitude=1e-2, seed=5)

    def setup(g):
        for nm, a in zip("UVWP", f):
            g.set(nm, a)
        g.connect(0, 2, "U", "V", "W", "P", corners=True)
        g.bound_flow()

    _same(*(_mixed(gpu_lib, case, ("mx_flux", v), setup) for v in (0, 1)))


@pytest.mark.parametrize("n", [12, 11])
def test_tiles_match_the_cell_order_around_a_body(gpu_lib, n):
    """The couplings a body closes, by masks in the pre-pass and the outer step."""
    case = cases.periodic_box(2, 1, 1, n=n, length=(2.0, 1.0, 1.0))
    bp, lists = cases.block_body(case, (6, 6, 6), (9, 8, 9), seed=7)

    def setup(g):
        load(g, case, bp, lists, random_fields(case, 3))
        g.connect(0, 2, "U", "V", "W", "P", corners=True)
        g.setpointvalues(True)

    _same(*(_mixed(gpu_lib, case, force, setup) for force in (None, ("mx_sip_sweep", 0))))


def test_tiles_match_the_cell_order_on_a_hierarchy_with_closed_cells(gpu_lib):
    """The table of the PAR blocks with BP: blocks with some, most and all of their
    cells closed next to a PAR face."""
    case, bp, lists = gc_hierarchy()
    bp = bp.copy()
    rng = np.random.default_rng(3)
    for g in _fine(case):
        B = _g3(case, bp, g)[2:-2, 2:-2, 2:-2]
        B[rng.random(B.shape) < 0.1] = 0.0
        B[:2, :4, :2] = 0.0
        B[-2:, -2:, 2:5] = 0.0
    f = np.random.default_rng(8)
    fields = {n: 0.1 * f.standard_normal(case.idim3d) for n in "UVW"}

    def setup(g):
        load_gc(g, case, bp, lists, fields)
        for lvl in (1, 2):
            g.connect(lvl, 2, v1="U", v2="V", v3="W", s1="P", corners=True)
        prepare_levels(g, case)
        g.setpointvalues(True)

    _same(*(_mixed(gpu_lib, case, force, setup) for force in (None, ("mx_sip_sweep", 0))))
