"""The ways a step reaches the GPU give the same bits: launch by launch (the
first two steps of a solver, and every one without graphs), as graph replays,
and as one chain of launches without side branches or early launches, which is
how a step is profiled.  Grids of whole transform planes, of line passes, and
one too large for early launches."""

import ctypes

import numpy as np
import pytest

from pllcart3d_b200 import _lib
from pllcart3d_b200.ic import workload_fields
from pllcart3d_b200.params import workload

pytestmark = pytest.mark.gpu

FIELDS = ("c_new", "u_new", "v_new", "w_new", "phi", "u_pg", "c_hn")
STEPS = 6


def _chain(s, n):
    k = 64
    names, ms, cnt, nk = ctypes.create_string_buffer(32 * k), (ctypes.c_double * k)(), (ctypes.c_int * k)(), ctypes.c_int()
    assert _lib.lib().pllgpu_profile_steps(s._h, n, k, names, ms, cnt, ctypes.byref(nk)) == 0


@pytest.mark.parametrize("precision", ["fp64", "mixed64", "mixed"])
@pytest.mark.parametrize("grid", ["64x32x32", "37x21x19", "20x128x128", "160x120x112"])
def test_same_bits_by_every_route(grid, precision):
    from pllcart3d_b200.solver import Solver

    wl = workload(f"fingering-{grid}")
    ic = workload_fields(wl)
    routes = {"graph": (True, [STEPS]), "one by one": (True, [1] * STEPS), "two at a time": (True, [2] * (STEPS // 2)),
              "stream": (False, [STEPS]), "chain": (False, None)}
    ref = None
    for name, (graph, calls) in routes.items():
        s = Solver(wl.params, precision=precision, use_graph=graph)
        s.load_ic(ic)
        if calls is None:
            _chain(s, STEPS)
        else:
            for n in calls:
                s.step(n)
        out = {f: s.get(f) for f in FIELDS}
        out["t"] = s.tval
        s.close()
        ref = ref or out
        for f in out:
            assert np.array_equal(out[f], ref[f]), (name, f)
