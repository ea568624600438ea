"""One entry that is not finite, wherever it stands in the block, ends in status -2, in every kernel that
reduces blocks, and the blocks beside it are solved."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,count", [(12, 3), (40, 5), (64, 400), (100, 1), (170, 400), (230, 3), (240, 528), (480, 2), (700, 2)])
@pytest.mark.parametrize("x", [float("nan"), float("inf")])
def test_status(n, count, x):
    import torch

    import nrgljubljana_b200 as nb
    g = torch.Generator(device="cuda").manual_seed(n)
    for i, j in ((0, 0), (0, 1), (0, n // 2), (n // 3, n - 1), (n - 3, n - 1), (n - 2, n - 1), (n - 1, n - 1)):
        H = [torch.triu(torch.randn(n, n, generator=g, device="cuda", dtype=torch.float64)) for _ in range(count)]
        E = [torch.empty(n, dtype=torch.float64, device="cuda") for _ in H]
        V = [torch.empty_like(h) for h in H]
        H[-1][i, j] = x
        info = nb.diag_batch_device(H, E, V)
        assert info[-1] == -2, (i, j)
        assert (info[:-1] == 0).all()
        assert all(torch.isfinite(e).all() for e in E[: min(3, count - 1)])
