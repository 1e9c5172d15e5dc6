"""Calls of the network library that are refused."""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, -1])
def test_loss_over_no_terms_is_refused(n):
    import torch

    from pllcart3d_b200 import surrogate as S

    a = torch.ones(4, device="cuda")
    loss = torch.zeros(1, device="cuda")
    assert S.nnlib().pllnn_mse(S._p(a), S._p(a), n, 1.0, None, S._p(loss), S._stream()) == 2
    assert S.nnlib().pllnn_mse(S._p(a), S._p(a), 4, 1.0, None, S._p(loss), S._stream()) == 0
