"""The batched explicit operator's tensor maps: ensembles built one after the
other, whose argument tables may lie where an earlier one's did, and classes of
every size that a launch's parameters hold maps for."""

import numpy as np
import pytest

from pllcart3d_b200.ic import workload_fields
from pllcart3d_b200.params import Workload, workload

pytestmark = pytest.mark.gpu

FIELDS = ("c_new", "u_new", "v_new", "w_new", "phi")


def _members(grid, n):
    base = workload("fingering-64x32x32").params
    p = base.replace(Nx_cell_global=grid[0], Ny_cell_global=grid[1], Nz_cell_global=grid[2])
    return [Workload(f"m{m}", p.replace(Vratio=-1.0 - 0.04 * m, Re=200.0 + 10 * m), modes=8, amplitude=0.01, seed=50 + m)
            for m in range(n)]


def _single(w, precision, steps):
    from pllcart3d_b200.solver import Solver

    s = Solver(w.params, precision=precision)
    s.load_ic(workload_fields(w))
    s.step(steps)
    return s


@pytest.mark.parametrize("precision", ["fp64", "mixed64", "mixed"])
def test_rebuilt_tables(precision):
    from pllcart3d_b200.ensemble import Ensemble

    # the same number of members and launches each time, so that the tables
    # have one size and the allocator hands out one address; other fields
    for grid in ((32, 16, 16), (24, 16, 16), (32, 16, 32), (16, 32, 16)):
        wls = _members(grid, 3)
        ens = Ensemble(wls, precision=precision)
        ens.load_ics()
        ens.step(2)
        ens.set_batching(2)   # and rebuilt within one ensemble
        ens.step(1)
        ens.set_batching(True)
        ens.step(2)
        for m, w in zip(ens.members, wls):
            s = _single(w, precision, 5)
            for f in FIELDS:
                assert np.array_equal(m.get(f), s.get(f)), (grid, w.name, f)
            s.close()
        ens.close()


# the class sizes at which a launch's tensor maps change form: 8 | 9, 40 | 41
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [8, 9, 41])
def test_class_sizes(n, precision):
    from pllcart3d_b200.ensemble import Ensemble

    wls = _members((16, 8, 8), n)
    ens = Ensemble(wls, precision=precision)
    ens.load_ics()
    ens.step(3)
    assert ens.classes == 1
    for m, w in zip(ens.members, wls):
        s = _single(w, precision, 3)
        for f in FIELDS:
            assert np.array_equal(m.get(f), s.get(f)), (w.name, f)
        s.close()
    ens.close()
