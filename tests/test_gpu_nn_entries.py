"""Entry points of the network library that the network itself does not call,
and calls that are refused."""

import numpy as np
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


# channel counts that go in 16-byte pieces and ones that go singly
@pytest.mark.parametrize("ca,cb", [(16, 8), (8, 24), (12, 4), (5, 3), (1, 16)])
def test_concatenate(ca, cb):
    import torch

    from pllcart3d_b200 import surrogate as S

    L, st, V = S.nnlib(), S._stream(), 77
    rng = np.random.default_rng(ca * 10 + cb)
    a = torch.tensor(rng.standard_normal((V, ca)), dtype=torch.bfloat16, device="cuda")
    b = torch.tensor(rng.standard_normal((V, cb)), dtype=torch.bfloat16, device="cuda")
    y = torch.zeros((V, ca + cb), dtype=torch.bfloat16, device="cuda")
    assert L.pllnn_cat_fwd(S._p(a), ca, S._p(b), cb, V, S._p(y), st) == 0
    assert torch.equal(y, torch.cat([a, b], 1))
    g = torch.tensor(rng.standard_normal((V, ca + cb)), dtype=torch.float32, device="cuda")
    da0 = torch.tensor(rng.standard_normal((V, ca)), dtype=torch.float32, device="cuda")
    db0 = torch.tensor(rng.standard_normal((V, cb)), dtype=torch.float32, device="cuda")
    for acc_a, acc_b in ((0, 1), (1, 0)):
        da, db = da0.clone(), db0.clone()
        assert L.pllnn_cat_bwd(S._p(g), ca, cb, V, S._p(da), acc_a, S._p(db), acc_b, st) == 0
        assert torch.equal(da, g[:, :ca] + (da0 if acc_a else 0))
        assert torch.equal(db, g[:, ca:] + (db0 if acc_b else 0))
    da = da0.clone()
    assert L.pllnn_cat_bwd(S._p(g), ca, cb, V, S._p(da), 0, None, 0, st) == 0   # one side alone
    assert torch.equal(da, g[:, :ca])
