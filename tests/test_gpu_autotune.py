"""The autotuner where its choices act (every variant of every kernel that has
variants gives the same bits) and where they do not (it leaves them alone)."""

import numpy as np
import pytest

from pllcart3d_b200.ic import workload_fields
from pllcart3d_b200.params import workload

pytestmark = pytest.mark.gpu

FIELDS = ("c_new", "u_new", "v_new", "w_new", "phi")

ACTS = [("32x16x16", dict(explicit_kernel="direct")), ("32x16x16", dict(exact_dct=True)),
        ("520x6x7", {}), ("6x520x7", {}), ("37x21x19", dict(explicit_kernel="direct", precision="mixed")),
        ("24x12x12", dict(exact_dct=True, precision="mixed")), ("520x6x7", dict(precision="mixed")),
        ("37x21x19", dict(explicit_kernel="direct", precision="mixed64"))]


def _solver(grid, kw):
    from pllcart3d_b200.solver import Solver

    wl = workload(f"fingering-{grid}")
    s = Solver(wl.params, **kw)
    s.load_ic(workload_fields(wl))
    return s


@pytest.mark.parametrize("grid,kw", ACTS)
def test_variants_that_act(grid, kw):
    ref = None
    for ve in range(4):
        for vl in range(3):
            s = _solver(grid, kw)
            s.set_tuning(ve, vl)
            s.step(3)
            out = {f: s.get(f) for f in FIELDS}
            s.close()
            ref = ref or out
            for f in FIELDS:
                assert np.array_equal(out[f], ref[f]), (ve, vl, f)
    # and the tuner's own choice, after as many steps
    s, t = _solver(grid, kw), _solver(grid, kw)
    t.step(s.autotune(1))
    assert np.array_equal(s.get("u_new"), t.get("u_new"))
    s.close()
    t.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed64", "mixed"])
def test_variants_that_do_not_act(precision):
    for keep in ((0, 1), (3, 2), (1, 0), (2, 2)):
        s, t = _solver("32x16x16", dict(precision=precision)), _solver("32x16x16", dict(precision=precision))
        s.set_tuning(*keep)
        done = s.autotune(1)
        assert done == 4 * 3 * 2
        assert s.tuning() == keep
        t.step(done)
        assert np.array_equal(s.get("u_new"), t.get("u_new"))
        s.close()
        t.close()
