"""Device memory of a solver: its state, one right-hand side and the Poisson
buffers; the sequential sweeps' scratch only where such a sweep runs."""

import pytest

from pllcart3d_b200.params import workload

pytestmark = pytest.mark.gpu

PAGE = 2 << 20   # the device allocates in pages of 2 MiB


# arrays of a padded field: 8 states, 8 convective terms, 8 viscosities, 3
# pressure gradients, phi, the divergence, a right-hand side and two Poisson
# buffers (the solves' other right-hand sides); the precision form's FP64
# staging field counts twice.  Past 512 rows in x the mode solve's scratch
# joins, past 512 in y or 256 in z the lines'.
@pytest.mark.parametrize("precision,grid,fields,exact", [
    ("fp64", (200, 128, 128), 32, False), ("mixed64", (200, 128, 128), 32, False), ("mixed", (200, 128, 128), 34, False),
    ("fp64", (96, 96, 300), 33, False), ("mixed", (24, 520, 200), 35, False),
    ("fp64", (600, 64, 64), 34, False), ("fp64", (200, 128, 128), 34, True)])
def test_memory_of_a_solver(precision, grid, fields, exact):
    import torch

    from pllcart3d_b200.solver import Solver

    p = workload("fingering-64x32x32").params.replace(Nx_cell_global=grid[0], Ny_cell_global=grid[1],
                                                      Nz_cell_global=grid[2])
    Solver(p, precision=precision, exact_dct=exact).close()   # the kernels are loaded
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    s = Solver(p, precision=precision, exact_dct=exact)
    used = before - torch.cuda.mem_get_info()[0]
    s.close()
    pitch = (grid[2] + 2 + 7) // 8 * 8
    field = (grid[0] + 6) * (grid[1] + 2) * pitch * (4 if precision == "mixed" else 8)
    # each array in whole pages, and 16 pages for everything of a line's or a
    # plane's size
    assert used <= fields * ((field + 1024 + PAGE - 1) // PAGE * PAGE) + 16 * PAGE, used / field
