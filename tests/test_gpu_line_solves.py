"""Whole steps against the CPU restatement on grids whose line lengths lie at
the edges of the partitioned solves' lane and row counts (4 .. 32 lanes of 8
rows, 32 of 16, the sequential sweeps beyond), along each axis, with odd and
even cross sections and partly filled tiles of neighbouring lines."""

import numpy as np
import pytest

from pllcart3d_b200.ic import cell_centres, workload_fields
from pllcart3d_b200.params import workload
from tests.util import rel_vector

pytestmark = pytest.mark.gpu

FIELDS = ("c_new", "u_new", "v_new", "w_new", "phi", "u_pg", "v_pg", "w_pg")

# (nx, ny, nz): one long axis each; the staggered components' lines are one
# row shorter, so each edge is met from both sides
GRIDS = [(4, 5, 4), (32, 9, 7), (33, 6, 20), (64, 7, 17), (65, 5, 33), (128, 5, 6), (129, 6, 5), (256, 4, 5),
         (257, 5, 4), (512, 4, 5), (513, 5, 4), (5, 32, 9), (6, 33, 16), (4, 65, 7), (5, 129, 6), (6, 256, 4),
         (4, 257, 5), (7, 6, 32), (5, 9, 33), (6, 5, 64), (5, 4, 65), (4, 7, 128), (6, 5, 129), (4, 5, 256),
         (5, 6, 257)]


def _smooth(p):
    """A smooth moving state: the ENO-2 closure picks the smaller of two
    second differences, so a saturated or two-valued c (or u = 1 throughout)
    lets rounding pick, and any two implementations part there."""
    xc, yc, zc = (a.reshape(sh) for a, sh in zip(cell_centres(p), ((-1, 1, 1), (1, -1, 1), (1, 1, -1))))
    sx, sy, sz = 2.0 * xc / p.X2, np.pi * (yc - p.Y1) / (p.Y2 - p.Y1), np.pi * (zc - p.Z1) / (p.Z2 - p.Z1)
    one = np.ones(p.shape)
    return {"c": 0.5 * (1.0 - np.tanh(sx - 1.0 - 0.1 * np.cos(sy) - 0.07 * np.cos(2.0 * sz))),
            "u": (1.0 + 0.1 * np.sin(1.3 * sx) * np.cos(sy + 0.3) + 0.04 * np.cos(sx + sz)) * one,
            "v": 0.08 * np.cos(1.1 * sx + 0.2) * np.sin(sy) * np.cos(sz + 0.4) * one,
            "w": 0.06 * np.cos(0.9 * sx - 0.3) * np.cos(sy + 0.5) * np.sin(sz) * one}


def _params(grid):
    """Cubic cells: stretched ones amplify the rounding of phi by 1/h^3 in the
    viscous part of the pressure gradient."""
    nx, ny, nz = grid
    return workload("fingering-%dx%dx%d" % grid).params.replace(
        X2=nx / 16.0, Y1=-ny / 32.0, Y2=ny / 32.0, Z1=-nz / 32.0, Z2=nz / 32.0)


def _run(grid, precision, steps):
    from oracle.pyref import OracleRun
    from pllcart3d_b200.solver import Solver

    p = _params(grid)
    ic = _smooth(p)
    o = OracleRun(p, ic)
    s = Solver(p, precision=precision)
    s.load_ic(ic)
    s.step(steps)
    o.steps(steps)
    assert s.status() == 0
    return {f: rel_vector(s.get, o.get, f) for f in FIELDS}


@pytest.mark.parametrize("grid", GRIDS, ids=lambda g: "x".join(map(str, g)))
def test_fp64_steps_at_line_length_edges(grid):
    errs = _run(grid, "fp64", 3)
    assert max(errs.values()) <= 1e-10, errs


# One substep's concentration, momentum and mode solves in the precision form
# against its sequential sweeps (exact_dct) from the same state: the explicit
# operators are the same kernel on the same values, so only the solves differ.
# Each of the three sweeps per variable has an inverse of norm <= 1 and rounds
# a row's coefficients and eliminated value in about 8 operations:
# 3 x 8 x 6e-8 = 1.4e-6 of the solution's increment.
@pytest.mark.parametrize("grid", GRIDS, ids=lambda g: "x".join(map(str, g)))
def test_fp32_solves_at_line_length_edges(grid):
    from pllcart3d_b200.solver import Solver

    p = _params(grid)
    ic = _smooth(p)
    runs = []
    for exact in (False, True):
        s = Solver(p, precision="mixed", exact_dct=exact)
        s.load_ic(ic)
        dt, g, r = 0.5 * s.find_cfl(), 8.0 / 15.0, 0.0
        vb = s.bulk_velo()
        s.concentration(dt, g, r, vb)
        s.calculate_viscosity()
        s.xmom(dt, g, r, vb)
        s.ymom(dt, g, r, vb)
        s.zmom(dt, g, r, vb)
        assert s.status() == 0
        runs.append(s)
    for f in ("c_new", "u_new", "v_new", "w_new"):
        assert rel_vector(runs[0].get, runs[1].get, f) <= 2e-6, f


def test_same_bits_on_every_run():
    """Warps that share lines with empty lanes, and the data-dependent end of
    the cyclic reduction, leave no room for run-to-run differences."""
    from pllcart3d_b200.solver import Solver

    wl = workload("fingering-37x21x19")
    ic = workload_fields(wl)
    out = []
    for _ in range(2):
        s = Solver(wl.params)
        s.load_ic(ic)
        s.step(4)
        out.append({f: s.get(f) for f in FIELDS})
    for f in FIELDS:
        assert np.array_equal(out[0][f], out[1][f]), f
