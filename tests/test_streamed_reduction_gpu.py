"""Batches whose reductions run on several kernels side by side: groups of CTAs, clusters, the
streaming kernel (two CTAs per SM) and the one-CTA kernel, with the streaming kernel at the
edges of its 8-column groups, 16-column panels and 64-row slabs and of the copies that its
shared memory holds."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(nb, sizes, seed, scale=1.0):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    H, E, V, H0 = [], [], [], []
    for n in sizes:
        a = torch.randn(n, n, generator=g, device="cuda", dtype=torch.float64) * scale
        h = torch.triu(a + a.T)
        H0.append(h.clone())
        H.append(h)
        E.append(torch.empty(n, dtype=torch.float64, device="cuda"))
        V.append(torch.empty(n, n, dtype=torch.float64, device="cuda"))
    info = nb.diag_batch_device(H, E, V)
    torch.cuda.synchronize()
    assert (info == 0).all()
    for h, e, v in zip(H0, E, V):
        n = h.shape[0]
        Hf = h + torch.triu(h, 1).T
        nrm = e.abs().max().item()
        assert (e[1:] >= e[:-1]).all()
        assert torch.linalg.norm(v @ Hf - e[:, None] * v, dim=1).max().item() <= 1e-12 * nrm * math.sqrt(n), n
        assert (v @ v.T - torch.eye(n, dtype=torch.float64, device="cuda")).abs().max().item() < 1e-10, n


@pytest.fixture(scope="module")
def nb():
    import nrgljubljana_b200 as m
    return m


@pytest.mark.parametrize("lo,hi,count", [(225, 290, 528), (440, 460, 420), (600, 641, 410)])
def test_edges(nb, lo, hi, count):
    """Every order of [lo, hi), enough blocks that they stream."""
    _check(nb, [lo + i % (hi - lo) for i in range(count)], 11)


def test_two_copies(nb):
    """Blocks whose product has two copies per CTA: orders where four leave no room for two CTAs."""
    _check(nb, [1700 + 7 * (i % 5) for i in range(8)] + [1601] * 330, 12)


@pytest.mark.parametrize("scale", [1e-150, 1e140])
def test_all_kernels_at_once(nb, scale):
    sizes = [1500, 1400] + [601 + 3 * (i % 20) for i in range(30)] + [230 + 11 * (i % 30) for i in range(300)]
    _check(nb, sizes + [20 + 5 * (i % 40) for i in range(200)], 13, scale)
