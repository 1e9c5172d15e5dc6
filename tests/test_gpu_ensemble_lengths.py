"""Ensembles whose grids differ in their folded transforms' lengths, the longer
ones first: one kernel serves every length with shared memory to match, so a
shorter length's launch must not take from a longer one's."""

import numpy as np
import pytest

from pllcart3d_b200.ic import workload_fields
from pllcart3d_b200.params import Workload, workload

pytestmark = pytest.mark.gpu

FIELDS = ("c_new", "u_new", "v_new", "w_new", "phi")

# classes of two below the default limit of shared memory, classes of two and
# single members above it (160 values and more), along y and along z
GRIDS = [
    [(24, 12, 12), (24, 12, 12), (16, 8, 8), (16, 8, 8)],
    [(8, 300, 8), (8, 300, 8), (8, 200, 8), (8, 200, 8)],
    [(8, 8, 300), (8, 8, 200)],
    [(8, 300, 8), (8, 12, 12), (8, 200, 8), (8, 12, 12)],
]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("grids", GRIDS)
def test_descending_lengths(grids, precision):
    from pllcart3d_b200.ensemble import Ensemble
    from pllcart3d_b200.solver import Solver

    base = workload("fingering-64x32x32").params
    wls = [Workload(f"m{m}", base.replace(Nx_cell_global=g[0], Ny_cell_global=g[1], Nz_cell_global=g[2],
                                          Vratio=-1.0 - 0.3 * m), modes=8, amplitude=0.01, seed=70 + m)
           for m, g in enumerate(grids)]
    ens = Ensemble(wls, precision=precision)
    ens.load_ics()
    ens.step(3)
    for m, w in zip(ens.members, wls):
        s = Solver(w.params, precision=precision)
        s.load_ic(workload_fields(w))
        s.step(3)
        for f in FIELDS:
            assert np.array_equal(m.get(f), s.get(f)), (w.name, f)
        s.close()
    ens.close()
