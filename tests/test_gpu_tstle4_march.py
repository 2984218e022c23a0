"""tstle4 of connected grids with one value of G (each face flux computed once, by
the cell before the face) against the oracle, bit for bit: cuts into several rows
and planes, rows of a few and of hundreds of cells, graded spacing, and values where
its exact halvings and corrected quotients leave the ordinary range; grids with a
value that is not finite or with several values of G go the general way."""
import numpy as np
import pytest

from mglet_gb300 import abi, cases

pytestmark = pytest.mark.gpu


def _compare(gpu_lib, oracle_lib, case, special=False, force=False):
    prm = abi.make_flow_params(gmol=1e-3, rho=1.3, gradp=(0.3, -0.2, 0.1), form=abi.FORM_PLAIN)
    pair = gpu_lib.Solver(case, prm), oracle_lib.Oracle(case, prm)
    rng = np.random.default_rng(3)
    n = case.idim3d // case.ngrid
    for nm in "UVWP":
        a = rng.standard_normal(case.idim3d)
        if special:
            a[rng.random(a.size) < 0.2] = 0.0
            a[rng.random(a.size) < 0.1] *= -0.0
            for scale in (1e-310, 1e-200, 1e-155, 1e140):
                a[rng.random(a.size) < 0.02] *= scale
            if nm in "UP":
                a[n + n // 2] = np.inf
                a[2 * n + n // 2] = np.nan
        for s in pair:
            s.set(nm, a)
    if special:
        G = np.full(case.idim3d, 1e-3)
        G[:n] += 1e-4 * rng.random(n)
        for s in pair:
            s.set("G", G)
    for s in pair:
        if force:
            f = np.random.default_rng(4)
            s.set_body_force(*(f.standard_normal(case.idim3d) for _ in range(3)))
        with np.errstate(all="ignore"):
            s.tstle4()
    for nm in ("UO", "VO", "WO"):
        assert np.array_equal(pair[0].get(nm), pair[1].get(nm), equal_nan=True), nm
    pair[0].close()


@pytest.mark.parametrize("tiles,shape", [
    ((1, 1, 1), (2, 2, 2)), ((2, 1, 1), (2, 3, 2)), ((2, 1, 2), (5, 40, 30)), ((1, 2, 1), (4, 3, 317)),
    ((1, 1, 1), (3, 2, 330)), ((3, 3, 2), (24, 24, 24)), ((6, 5, 6), (13, 9, 11))])
def test_march_bit_exact(gpu_lib, oracle_lib, tiles, shape):
    ni, nj, nk = shape
    _compare(gpu_lib, oracle_lib, cases.stretch(cases.periodic_box(*tiles, n=ni, nj=nj, nk=nk)))


def test_march_special_values(gpu_lib, oracle_lib):
    _compare(gpu_lib, oracle_lib, cases.periodic_box(2, 2, 1, n=12), special=True)


def test_march_body_force_and_walls(gpu_lib, oracle_lib):
    walls = {3: abi.BC_FIX, 4: abi.BC_SLI}   # (the wall function's pow is not the oracle's to the bit)
    _compare(gpu_lib, oracle_lib, cases.periodic_box(2, 3, 2, n=8, walls=walls), force=True)
