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


# channel counts that go in 16-byte pieces and ones that go singly
@pytest.mark.parametrize("ca,cb", [(16, 8), (64, 32), (12, 4), (5, 3), (8, 0)])
def test_upsample_concatenate(ca, cb):
    import torch

    from pllcart3d_b200 import surrogate as S

    L, st = S.nnlib(), S._stream()
    vol = (2, 3, 2, 5)
    fine = (2, 6, 4, 10)
    rng = np.random.default_rng(ca * 10 + cb)
    a, b = _bf16(rng.standard_normal(vol + (ca,))), _bf16(rng.standard_normal(fine + (cb,)))
    ad, bd = a.cuda().contiguous(), b.cuda().contiguous()
    y = torch.zeros(fine + (ca + cb,), dtype=torch.bfloat16, device="cuda")
    assert L.pllnn_upcat_fwd(S._p(ad), *vol, ca, S._p(bd), cb, S._p(y), st) == 0
    ref = np.concatenate([nn_ref.up(a.float().numpy()), b.float().numpy()], -1)
    assert np.array_equal(y.float().cpu().numpy(), ref)
    g = rng.standard_normal(fine + (ca + cb,)).astype(np.float32)
    start = rng.standard_normal(vol + (ca,)).astype(np.float32)
    gd, da = torch.tensor(g, device="cuda"), torch.tensor(start, device="cuda")
    db = torch.zeros(fine + (cb,), dtype=torch.float32, device="cuda")
    assert L.pllnn_upcat_bwd(S._p(gd), *vol, ca, cb, S._p(da), 1, S._p(db), st) == 0
    assert np.array_equal(db.cpu().numpy(), g[..., ca:])
    ref = start + nn_ref.up_bwd(g[..., :ca].astype(np.float64))
    # eight FP32 additions of the children and one of the start value
    assert np.all(np.abs(da.cpu().numpy() - ref) <= 9 * 2.0 ** -24 * (np.abs(start) + nn_ref.up_bwd(np.abs(g[..., :ca]))))


@pytest.mark.parametrize("c", [16, 6, 1])
def test_pooling(c):
    import torch

    from pllcart3d_b200 import surrogate as S

    L, st = S.nnlib(), S._stream()
    rng = np.random.default_rng(c)
    x = _bf16(rng.standard_normal((2, 4, 6, 2, c)))
    xd = x.cuda().contiguous()
    y = torch.zeros((2, 2, 3, 1, c), dtype=torch.bfloat16, device="cuda")
    assert L.pllnn_pool_fwd(S._p(xd), 2, 4, 6, 2, c, S._p(y), st) == 0
    ref = nn_ref.pool(x.double().numpy())
    # BF16 rounding of an FP32 mean
    assert np.all(np.abs(y.double().cpu().numpy() - ref) <= 2.0 ** -8 * np.abs(ref) + 1e-6)
    g = rng.standard_normal((2, 2, 3, 1, c)).astype(np.float32)
    gd, dx = torch.tensor(g, device="cuda"), torch.zeros((2, 4, 6, 2, c), dtype=torch.float32, device="cuda")
    assert L.pllnn_pool_bwd(S._p(gd), 2, 4, 6, 2, c, S._p(dx), 0, st) == 0
    assert np.array_equal(dx.cpu().numpy(), nn_ref.pool_bwd(g).astype(np.float32))
