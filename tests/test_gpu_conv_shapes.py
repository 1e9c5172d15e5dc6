"""The tcgen05 convolution and weight gradient against FP64 on the same BF16
inputs, at the shapes where their tiles can go wrong: boxes of fewer than 128
voxels, boxes past the volume's edge in h and d, w rows that do not divide a
tile, every channel group (16, 32, 64), column counts of 16 to 256 and 96,
row tiles filled by part of a tap's channels or by several taps, and voxel
tiles fewer than the CTAs."""

import numpy as np
import pytest

from oracle import nn_ref

pytestmark = pytest.mark.gpu

SHAPES = [
    (3, 16, 32, (1, 8, 16, 64)), (3, 96, 32, (1, 4, 6, 64)), (3, 32, 96, (1, 3, 4, 64)), (3, 32, 64, (2, 5, 7, 56)),
    (3, 64, 128, (1, 3, 5, 14)), (3, 128, 256, (1, 4, 5, 7)), (3, 384, 128, (1, 2, 3, 16)),
    (3, 192, 64, (1, 4, 4, 32)), (3, 64, 192, (1, 6, 10, 12)), (1, 32, 16, (1, 4, 8, 64)), (3, 16, 16, (1, 1, 1, 128)),
    (3, 32, 32, (1, 1, 3, 1)), (3, 48, 80, (2, 2, 3, 50)), (1, 16, 48, (1, 2, 2, 130)), (3, 16, 32, (1, 2, 3, 129)),
]


def _bf16(a):
    import torch

    return torch.tensor(a, dtype=torch.float32).to(torch.bfloat16)


def _inputs(k, ci, co, vol):
    rng = np.random.default_rng(ci * 1000 + co + vol[3])
    x = _bf16(rng.standard_normal(vol + (ci,)))
    w = _bf16(rng.standard_normal((co, k ** 3, ci)) / np.sqrt(k ** 3 * ci))
    g = _bf16(rng.standard_normal(vol + (co,)))
    return x, w, g


# FP32 accumulation of exact BF16 products, 16 at a time: every addition rounds
# (or truncates) at 2^-23 of the running sum, which the sum of the products'
# magnitudes bounds
def _bound(terms, magnitude):
    return 2.0 ** -23 * (terms / 16 + 8) * magnitude


@pytest.mark.parametrize("k,ci,co,vol", SHAPES)
def test_forward(k, ci, co, vol):
    import torch

    from pllcart3d_b200 import surrogate as S

    x, w, _ = _inputs(k, ci, co, vol)
    V = int(np.prod(vol))
    xd, wd = x.cuda().contiguous(), w.cuda().contiguous()
    z = torch.full((V, co), float("nan"), dtype=torch.float32, device="cuda")
    assert S.nnlib().pllnn_conv_fwd(S._p(xd), *vol, ci, S._p(wd), None, co, k, S._p(z), None, 0, 0.0, S._stream()) == 0
    torch.cuda.synchronize()
    assert S.nnlib().pllnn_status() == 0
    xf, wf = x.double().numpy(), w.double().numpy()
    ref = nn_ref.conv_fwd(xf, wf, None, k).reshape(V, co)
    mag = nn_ref.conv_fwd(np.abs(xf), np.abs(wf), None, k).reshape(V, co)
    assert np.all(np.abs(z.cpu().numpy() - ref) <= _bound(k ** 3 * ci, mag))


@pytest.mark.parametrize("k,ci,co,vol", SHAPES)
def test_weight_gradient(k, ci, co, vol):
    import torch

    from pllcart3d_b200 import surrogate as S

    x, w, g = _inputs(k, ci, co, vol)
    xd, gd = x.cuda().contiguous(), g.cuda().contiguous()
    start = torch.tensor(np.random.default_rng(3).standard_normal(w.shape), dtype=torch.float32)
    dw = start.cuda().contiguous()
    assert S.nnlib().pllnn_conv_wgrad(S._p(gd), S._p(xd), *vol, ci, co, k, S._p(dw), S._stream()) == 0
    torch.cuda.synchronize()
    assert S.nnlib().pllnn_status() == 0
    xf, wf, gf = x.double().numpy(), w.double().numpy(), g.double().numpy()
    ref = nn_ref.conv_bwd(xf, wf, gf, k)[1] + start.double().numpy()
    mag = nn_ref.conv_bwd(np.abs(xf), wf, np.abs(gf), k)[1] + np.abs(start.numpy())
    assert np.all(np.abs(dw.cpu().numpy() - ref) <= _bound(int(np.prod(vol)), mag))
