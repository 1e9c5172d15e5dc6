"""The precision form's sequential mode solve, for lines longer than the
partitioned one takes, against the FP64 form's on the same divergence: line
lengths around its blocks of 16 rows, planes of the line passes and of the
tcgen05 ones (modes stored the other way round)."""

import numpy as np
import pytest

from pllcart3d_b200.params import workload

pytestmark = pytest.mark.gpu


# Five FP32 roundings (right-hand side, three passes, phi: 6e-8 each of the
# array's largest value) of a field whose lowest mode the inverse amplifies no
# more than ten times as much as its highest one
TOL = 5 * 6e-8 * 10


@pytest.mark.parametrize("grid", [(513, 6, 9), (527, 8, 12), (528, 5, 7), (529, 12, 10), (1024, 20, 6), (520, 128, 128)],
                         ids=lambda g: "x".join(map(str, g)))
def test_long_lines(grid):
    from pllcart3d_b200.solver import Solver

    nx, ny, nz = grid
    p = workload("fingering-%dx%dx%d" % grid).params.replace(X2=nx / 16.0, Y1=-ny / 32.0, Y2=ny / 32.0, Z1=-nz / 32.0,
                                                             Z2=nz / 32.0)
    x, y, z = ((np.arange(n) + 0.5) / n for n in grid)
    div = np.zeros(p.shape)
    div[3:nx + 3, 1:ny + 1, 1:nz + 1] = (
        np.cos(np.pi * x)[:, None, None] + 0.5 * np.cos(3 * np.pi * x)[:, None, None] * np.cos(np.pi * y)[:, None]
        + 0.4 * np.cos(2 * np.pi * x)[:, None, None] * np.cos(np.pi * z))
    phi = []
    for precision in ("mixed", "fp64"):
        s = Solver(p, precision=precision)
        s.set("div", div)
        s.phisolver_dct(0.01, 1.0, 0.0)
        phi.append(s.get("phi")[3:nx + 3, 1:ny + 1, 1:nz + 1])
        s.close()
    assert np.abs(phi[0] - phi[1]).max() <= TOL * np.abs(phi[1]).max()
