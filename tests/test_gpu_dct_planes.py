"""Whole steps on grids whose y-z planes are transformed whole (sides of 32,
64 and 128 points, up to 4096 of them) and just past that, against the CPU restatement, and phi's
ghost points, which the inverse transform writes, in both forms."""

import numpy as np
import pytest

from tests.test_gpu_line_solves import _params, _run, _smooth

pytestmark = pytest.mark.gpu

SIDES = (32, 64, 128)
PLANES = [(ny, nz) for ny in SIDES for nz in SIDES]


# the tolerance of the line-length test: the same smooth state, cubic cells
# and three steps, with transforms whose error grows as log n
@pytest.mark.parametrize("ny,nz", PLANES)
def test_fp64_steps_on_whole_planes(ny, nz):
    errs = _run((5, ny, nz), "fp64", 3)
    assert max(errs.values()) <= 1e-10, errs


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("grid", [(4, 32, 64), (9, 64, 32)], ids=lambda g: "x".join(map(str, g)))
def test_phi_ghost_points(grid, precision):
    from pllcart3d_b200.solver import Solver

    p = _params(grid)
    s = Solver(p, precision=precision)
    s.load_ic(_smooth(p))
    s.step(1)
    phi, (nx, ny, nz) = s.get("phi"), grid
    i, j, k = slice(3, nx + 3), slice(1, ny + 1), slice(1, nz + 1)
    assert np.any(phi[i, j, k])
    for ghost, cell in (((2, j, k), (3, j, k)), ((nx + 3, j, k), (nx + 2, j, k)), ((i, 0, k), (i, 1, k)),
                        ((i, ny + 1, k), (i, ny, k)), ((i, j, 0), (i, j, 1)), ((i, j, nz + 1), (i, j, nz))):
        assert np.array_equal(phi[ghost], phi[cell])
