"""A launch that the runtime refuses while a step's graph is built is an error
of the call, not a step without that kernel.  The exact form's flux sums keep
two values per y row in shared memory and take no more than the default 48 KB,
so a line of 3100 rows is refused on the host."""

import ctypes

import pytest

from pllcart3d_b200 import _lib
from pllcart3d_b200.ic import workload_fields
from pllcart3d_b200.params import Workload, workload
from pllcart3d_b200.solver import Solver

pytestmark = pytest.mark.gpu

ECUDA = 2


def _run():
    p = workload("fingering-64x32x32").params.replace(Nx_cell_global=4, Ny_cell_global=3100, Nz_cell_global=4)
    return p, workload_fields(Workload("tall", p, modes=8, amplitude=0.01, seed=5))


def test_single_run():
    p, ic = _run()
    for graph in (False, True):
        s = Solver(p, exact_dct=True, use_graph=graph)
        s.load_ic(ic)
        for _ in range(3):
            with pytest.raises(_lib.PllGpuError) as e:
                s.step(1)
            assert e.value.code == ECUDA
        s.close()


def test_ensemble():
    p, ic = _run()
    L = _lib.lib()
    cp = Solver.c_params(p, exact_dct=True)
    h = ctypes.c_void_p(L.pllgpu_ensemble_create(1, ctypes.byref(cp), 0))
    assert h
    v = Solver.view(L.pllgpu_ensemble_member(h, 0), p, "fp64")
    for k in "cuvw":
        v.set(f"{k}_new", ic[k])
    assert L.pllgpu_ensemble_start(h) == 0
    assert L.pllgpu_ensemble_steps(h, 1) == ECUDA
    L.pllgpu_ensemble_destroy(h)
