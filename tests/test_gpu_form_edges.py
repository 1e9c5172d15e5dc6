"""One step of mixed64 against the FP64 form at the line lengths and on the planes
where the solves and transforms change form."""

import pytest

from tests.test_gpu_dct_planes import PLANES
from tests.test_gpu_line_solves import GRIDS, _params, _smooth
from tests.util import rel_vector

pytestmark = pytest.mark.gpu

# the WENO5 weights carry about 10 roundings of 6e-8 into a correction of at
# most a cell's difference (0.2), three axes, half a cell's travel: 2e-7
TOL = 1e-6


@pytest.mark.parametrize("grid", GRIDS + [(5, *p) for p in PLANES] + [(4, 128, 128), (6, 256, 128)],
                         ids=lambda g: "x".join(map(str, g)))
def test_one_step(grid):
    from pllcart3d_b200.solver import Solver

    p = _params(grid)
    ic = _smooth(p)
    runs = []
    for form in ("mixed64", "fp64"):
        s = Solver(p, precision=form)
        s.load_ic(ic)
        s.step(1)
        assert s.status() == 0
        runs.append(s)
    errs = {f: rel_vector(runs[0].get, runs[1].get, f) for f in ("c_new", "u_new", "v_new", "w_new")}
    for s in runs:
        s.close()
    assert max(errs.values()) <= TOL, errs
