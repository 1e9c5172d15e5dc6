"""The weight gradient on volumes at the edges of the rule that takes small ones
to the warp-level kernel (64 voxels; for 3x3x3 kernels 96, and 160 from 32 channels
on), against FP64 on the same BF16 inputs."""

import numpy as np
import pytest

from oracle import nn_ref
from tests.test_gpu_conv_shapes import _bound, _inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,ci,co", [(3, 16, 32), (3, 32, 32), (3, 64, 48), (1, 32, 64)])
@pytest.mark.parametrize("vol", [(1, 1, 1, 1), (1, 2, 2, 2), (1, 3, 3, 7), (1, 4, 4, 4), (1, 5, 19, 1), (1, 4, 4, 6),
                                 (1, 3, 53, 1), (1, 5, 4, 8), (2, 4, 4, 5)])
def test_small_volumes(k, ci, co, vol):
    import torch

    from pllcart3d_b200 import surrogate as S

    x, w, g = _inputs(k, ci, co, vol)
    xd, gd = x.cuda().contiguous(), g.cuda().contiguous()
    dw = torch.zeros(w.shape, dtype=torch.float32, device="cuda")
    assert S.nnlib().pllnn_conv_wgrad(S._p(gd), S._p(xd), *vol, ci, co, k, S._p(dw), S._stream()) == 0
    torch.cuda.synchronize()
    assert S.nnlib().pllnn_status() == 0
    xf, wf, gf = x.double().numpy(), w.double().numpy(), g.double().numpy()
    ref = nn_ref.conv_bwd(xf, wf, gf, k)[1]
    mag = nn_ref.conv_bwd(np.abs(xf), wf, np.abs(gf), k)[1]
    assert np.all(np.abs(dw.cpu().numpy() - ref) <= _bound(int(np.prod(vol)), mag))
