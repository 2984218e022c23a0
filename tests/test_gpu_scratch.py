"""Contexts on a device without room for what they can do without: tables and arrays
of the solves on tiles, the table of the PAR blocks.  They take the kernels that need
less, with the same bits, and give back what they had taken."""
import numpy as np
import pytest

from mglet_gb300 import abi, cases
from test_oracle_gc_levels import gc_hierarchy, load_gc
from test_oracle_ghostcell import gc_case, load, random_fields
from test_oracle_levels import prepare_levels

pytestmark = pytest.mark.gpu


@pytest.fixture
def limit(gpu_lib):
    yield gpu_lib.load().mglet_gpu_test_scratch_limit
    gpu_lib.load().mglet_gpu_test_scratch_limit(-1)


def _graded():
    return cases.stretch(cases.periodic_box(3, 2, 2, n=10, nj=9, nk=8, length=(2.0, 2.0, 1.0),
                                            walls={1: abi.BC_FIX, 2: abi.BC_OP1, 3: abi.BC_NOS}))


def _one_level(g, case):
    for nm, a in zip("UVWP", cases.add_noise(case, cases.taylor_green(case), seed=5)):
        g.set(nm, a)
    g.connect(0, 2, "U", "V", "W", "P", corners=True)
    g.bound_flow()


def _body(g, case):
    _, bp, lists = gc_case(seed=7)
    load(g, case, bp, lists, random_fields(case, 3))
    g.connect(0, 2, "U", "V", "W", "P", corners=True)
    g.setpointvalues(True)


def _levels(g, case):
    _, bp, lists = gc_hierarchy()
    f = np.random.default_rng(8)
    load_gc(g, case, bp, lists, {n: 0.1 * f.standard_normal(case.idim3d) for n in "UVW"})
    for lvl in (1, 2):
        g.connect(lvl, 2, v1="U", v2="V", v3="W", s1="P", corners=True)
    prepare_levels(g, case)
    g.setpointvalues(True)


def _run(gpu_lib, case, form, setup, left, limit):
    limit(left)
    g = gpu_lib.Solver(case, abi.make_flow_params(gmol=1e-2, epcorr=1e-12, nouter=3, ninner=3, form=form))
    setup(g, case)
    rk = gpu_lib.rk_scheme("williamson")
    n0 = g.launches
    st = [g.timeintegrate_flow(1, 1, 0.0, 2e-3, irk, rk) for irk in (1, 2, 3)]
    n, text = g.launches - n0, g.tuning()
    limit(-1)
    out = [g.get(nm) for nm in ("U", "V", "W", "P", "DP")]
    g.close()
    return n, text, [(s.nouter_done, s.maxrhs) for s in st], out


@pytest.mark.parametrize("case,form,setup", [
    (_graded, abi.FORM_PLAIN, _one_level), (_graded, abi.FORM_MIXED, _one_level),
    (lambda: gc_case(seed=7)[0], abi.FORM_MIXED, _body),
    (lambda: gc_hierarchy()[0], abi.FORM_MIXED, _levels)])
def test_the_smaller_path_gives_the_same_bits(gpu_lib, limit, case, form, setup):
    case = case()
    n, text, stats, fields = _run(gpu_lib, case, form, setup, -1, limit)
    ways = set()
    for left in range(26):
        m, t, s, f = _run(gpu_lib, case, form, setup, left, limit)
        assert s == stats, left
        for x, y in zip(f, fields):
            assert np.array_equal(x, y), left
        ways.add((m, "2x2x2 tiles" in t))
        if left == 0:
            assert "2x2x2 tiles" not in t and (m, t) != (n, text)
    assert (m, "2x2x2 tiles" in t) == (n, "2x2x2 tiles" in text)   # the last has all it asks for
    assert len(ways) >= (3 if setup is _levels else 2)


@pytest.mark.parametrize("call", ["set_ghostcell", "set_scalars", "energy_gradient", "set_body_force", "BP"])
def test_memory_goes_back_when_it_is_needed(gpu_lib, limit, call):
    """A plain context on tiles, and a call that ends the solve on tiles or needs
    memory itself when there is none: it gives the tiles' memory back and goes on."""
    import torch
    case = cases.periodic_box(4, 4, 4, n=16)
    kw = dict(gmol=1e-2, epcorr=0.0, nouter=3, ninner=3, nouter_min=3, form=abi.FORM_PLAIN)
    rk = gpu_lib.rk_scheme("williamson")

    def run(starved):
        g = gpu_lib.Solver(case, abi.make_flow_params(**kw))
        _one_level(g, case)
        free = torch.cuda.mem_get_info()[0]
        if starved:
            limit(0)
        out = []
        if call == "set_ghostcell":
            g.set_ghostcell()
            g.setpointvalues(True)
        elif call == "set_scalars":
            g.set_scalars([0.71])
        elif call == "BP":
            g.set("BP", np.ones(case.idim3d))
        else:
            g.set_body_force(*(np.full(case.idim3d, 0.1) for _ in range(3)))
            if call == "energy_gradient":
                out.append(g.energy_gradient(1, 1, 1e-3, rk)[0])
        used = free - torch.cuda.mem_get_info()[0]
        limit(-1)
        g.timeintegrate_flow(1, 1, 0.0, 1e-3, 1, rk)
        out += [g.get(nm) for nm in "UVWP"]
        g.close()
        return used, out

    (ua, a), (ub, b) = run(False), run(True)
    scratch = 6 * case.ncells * 8   # the arrays of the solve
    # (half of it: what the driver takes for itself goes either way)
    if call in ("set_ghostcell", "BP"):
        assert abs(ua - ub) < scratch // 2
    else:
        assert ua - ub > scratch // 2
    if call == "BP":
        assert ua < -scratch // 2
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
