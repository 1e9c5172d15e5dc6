"""The Poisson solve's whole-line DCT passes (FFT for powers of two, the folded
dense product otherwise, both storage types) against the CPU restatement, at
lengths around the 4-term, 8-output and 32-line groups of the folded product,
its longest line, mixed axes, and line counts that leave partly filled tiles."""

import numpy as np
import pytest

from pllcart3d_b200.params import workload
from tests.util import rel_maxnorm

pytestmark = pytest.mark.gpu

PLANES = [(4, 4), (5, 7), (6, 9), (7, 8), (15, 17), (16, 9), (31, 16), (33, 15), (32, 75), (53, 64), (90, 70), (64, 16),
          (127, 6), (128, 5), (6, 129), (5, 256), (255, 4), (4, 511), (512, 5), (513, 4), (5, 514)]


def _phi(plane, precision, nx=5):
    """phi of the same right-hand side, by the restatement and the GPU."""
    from oracle.pyref import OracleRun
    from pllcart3d_b200.ic import workload_fields
    from pllcart3d_b200.solver import Solver

    ny, nz = plane
    wl = workload(f"fingering-{nx}x{ny}x{nz}")
    p = wl.params.replace(X2=nx / 16.0, Y1=-ny / 32.0, Y2=ny / 32.0, Z1=-nz / 32.0, Z2=nz / 32.0)
    wl.params = p
    ic = workload_fields(wl)
    # a source whose values FP32 holds exactly, smooth and rough parts
    rng = np.random.default_rng(ny * 1000 + nz)
    i, j, k = np.meshgrid(*(np.arange(n) for n in p.shape), indexing="ij")
    div = (np.cos(0.7 * i) * np.cos(0.05 * j + 1.0) * np.sin(0.04 * k + 0.5) + 0.2 * rng.standard_normal(p.shape))
    div = div.astype(np.float32).astype(np.float64)
    out = []
    for s in (OracleRun(p, ic), Solver(p, precision=precision)):
        gpu = isinstance(s, Solver)
        if gpu:
            s.load_ic(ic)
            s.set("div", div)
            s.phisolver_dct(0.01, 8.0 / 15.0, 0.0)
        else:
            s.view("div")[...] = div
            s.call("phisolver", 0.01, 8.0 / 15.0, 0.0)
        out.append(s.get("phi")[3:-3, 1:-1, 1:-1])
    return out


@pytest.mark.parametrize("plane", PLANES, ids=lambda p: "x".join(map(str, p)))
def test_fp64_phi(plane):
    ref, got = _phi(plane, "fp64")
    assert rel_maxnorm(got, ref) <= 1e-11


# FP32 storage of the source and of the three intermediate arrays, FP64
# arithmetic: four roundings of 6e-8 of an array's largest value, each passed on
# by transforms whose normalised forms do not amplify
@pytest.mark.parametrize("plane", PLANES, ids=lambda p: "x".join(map(str, p)))
def test_fp32_phi(plane):
    ny, nz = plane
    ref, got = _phi(plane, "mixed")
    tol = 1e-6 if max(plane) <= 512 else 514 * 6e-8   # beyond: the split-TF32 product's FP32 sums
    assert rel_maxnorm(got, ref) <= tol
