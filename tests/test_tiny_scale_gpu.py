"""Blocks of very small and very large norm: the merges solve their secular equations in units
in which squares of eigenvector components and of pole distances stay in range."""
import math

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1e-150, 1e-140, 1e150])
@pytest.mark.parametrize("n", [50, 90, 230, 700])
def test_scaled_blocks(n, scale):
    import torch

    import nrgljubljana_b200 as nb
    g = torch.Generator(device="cuda").manual_seed(n)
    a = torch.randn(n, n, generator=g, device="cuda", dtype=torch.float64)
    h0 = torch.triu(a + a.T)
    e = torch.empty(n, dtype=torch.float64, device="cuda")
    v = torch.empty(n, n, dtype=torch.float64, device="cuda")
    assert (nb.diag_batch_device([h0 * scale], [e], [v]) == 0).all()
    torch.cuda.synchronize()
    Hf = h0 + torch.triu(h0, 1).T
    e = e / scale
    assert torch.linalg.norm(v @ Hf - e[:, None] * v, dim=1).max().item() <= 1e-12 * e.abs().max().item() * math.sqrt(n)
    assert (v @ v.T - torch.eye(n, dtype=torch.float64, device="cuda")).abs().max().item() < 1e-10
