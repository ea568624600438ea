"""Batches of blocks for the one-CTA solver: calls that the SMs hold at once (one launch) and larger ones (a
launch per class of order, up to 16, 32, 64, 96, where there are enough), at the edges of the classes,
alone and beside larger blocks."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("orders,count", [([1, 2, 16, 17, 32, 33, 64], 148), ([16, 17], 149), ([1, 16], 1000),
                                          ([64, 33, 32, 17, 16, 3], 1200), ([96, 65, 64, 33, 32, 16, 5], 1500),
                                          ([64, 16], 297), ([65, 64], 150), ([300, 16, 40], 900),
                                          ([33, 32], 1776), ([33, 32], 1778)])
def test_classes(orders, count):
    import torch

    import nrgljubljana_b200 as nb
    ctx = nb.Context()
    ctx.set_tuning(small_max_n=96)
    g = torch.Generator(device="cuda").manual_seed(count)
    H, E, V, H0 = [], [], [], []
    for i in range(count):
        n = orders[i % len(orders)]
        h = torch.triu(torch.randn(n, n, generator=g, device="cuda", dtype=torch.float64))
        H0.append(h.clone())
        H.append(h)
        E.append(torch.full((n,), float("nan"), dtype=torch.float64, device="cuda"))
        V.append(torch.full((n, n), float("nan"), dtype=torch.float64, device="cuda"))
    assert (nb.diag_batch_device(H, E, V, ctx=ctx) == 0).all()
    torch.cuda.synchronize()
    for i in np.random.default_rng(0).permutation(count)[:300]:
        h, e, v = H0[i], E[i], V[i]
        n = h.shape[0]
        Hf = h + torch.triu(h, 1).T
        assert (e[1:] >= e[:-1]).all()
        assert torch.linalg.norm(v @ Hf - e[:, None] * v, dim=1).max().item() <= 1e-12 * e.abs().max().item() * math.sqrt(n)
        assert (v @ v.T - torch.eye(n, dtype=torch.float64, device="cuda")).abs().max().item() < 1e-10
