"""Blocks in which numbers far below the block's norm matter: degenerate states coupled by next to
nothing, parts that are tiny beside the rest, matrices of low rank, against the oracle's dsyev."""
import numpy as np
import pytest

from eigcheck import check_eig

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nb():
    import nrgljubljana_b200 as m
    m.context()
    return m


def check_all(nb, oracle, blocks, **tuning):
    ctx = nb.Context()
    if tuning:
        ctx.set_tuning(**tuning)
    for h, g in zip(blocks, nb.diagonalisations(blocks, ctx=ctx, check_upper=False)):
        w, v = oracle.diagonalise(h)
        check_eig(h, g.val, g.vec, w, v, oracle)


def test_degenerate_pairs(nb, oracle):
    """Two states of energy zero coupled by t, at the end of a diagonal block and in the middle of a full one:
    every solver, and the leaves of the divide and conquer."""
    blocks = []
    for t in (1e-150, 1e-163, 1e-200, 1e-300):
        for n in (3, 9, 40, 64, 96, 300):
            h = np.diag(np.r_[1.0 / np.arange(1, n - 1), 0.0, 0.0])
            h[-2, -1] = t
            blocks.append(h)
            m = n // 2
            g = np.triu(np.random.default_rng(n).standard_normal((n, n)))
            g[m - 1:m + 1, :] = g[:, m - 1:m + 1] = 0.0
            g[m - 1, m] = t
            blocks.append(g)
    check_all(nb, oracle, blocks, small_max_n=96)


def test_smallest_norms(nb):
    for norm in (2.0 ** -1010, 2.0 ** -1022):
        got = nb.diagonalisations([norm * np.array([[1.0, 0.5], [0.0, 1.0]])])[0]
        assert np.abs(got.val / norm - [0.5, 1.5]).max() <= 1e-15 + 5e-324 / norm
        assert np.abs(got.vec @ got.vec.T - np.eye(2)).max() <= 1e-15


def test_tiny_tails(nb, oracle):
    """Blocks of order one whose last two thirds are a tridiagonal matrix of size x."""
    blocks = []
    for x in (1e-100, 1e-155, 1e-163, 1e-300):
        for n in (12, 20, 40, 64, 96, 300, 700):
            d, e = np.full(n, x), np.full(n, x)
            d[: n // 3], e[: n // 3] = 1.0 + np.arange(n // 3), 0.5
            blocks.append(np.diag(d) + np.diag(e[:-1], 1))
    check_all(nb, oracle, blocks, small_max_n=96)


def low_rank(n, kind, t=0.0):
    rng = np.random.default_rng(n)
    if kind == "constant":
        return np.triu(np.full((n, n), 0.3))
    if kind == "rank two":
        a = rng.standard_normal((n, 2))
        return np.triu(a @ a.T)
    h = np.triu(rng.standard_normal((n, n)))  # the first row's squares underflow
    h[0, 1:] *= t
    return h


def test_low_rank_one_cta(nb, oracle):
    blocks = [low_rank(n, kind) for n in range(2, 97) for kind in ("constant", "rank two")]
    blocks += [low_rank(n, "tiny column", t) for n in (3, 30, 64, 96) for t in (1e-135, 1e-157, 1e-160, 1e-250)]
    check_all(nb, oracle, blocks, small_max_n=96)


# one block: 16 CTAs in a cluster or a group of many; many: single CTAs, clusters of few
@pytest.mark.parametrize("n", [70, 128, 230, 449, 601, 900])
def test_low_rank_larger(nb, oracle, n):
    for kind, t in (("constant", 0.0), ("rank two", 0.0), ("tiny column", 1e-157), ("tiny column", 1e-161)):
        check_all(nb, oracle, [low_rank(n, kind, t)])
    check_all(nb, oracle, [low_rank(m, "constant") for m in (225, 226, 230, 301, 402, 300, 171, 165)])


@pytest.mark.parametrize("n,count", [(170, 400), (240, 528), (601, 410)])
def test_low_rank_in_large_batches(nb, n, count):
    """The kernels of large batches: one CTA's packed triangle (up to mid_max_n), the streaming reduction."""
    import torch
    H0 = [torch.tensor(low_rank(n + i % 3, kind, t), device="cuda")
          for i in range(3) for kind, t in (("constant", 0.0), ("rank two", 0.0), ("tiny column", 1e-157))]
    H = [H0[i % len(H0)].clone() for i in range(count)]
    E = [torch.empty(h.shape[0], dtype=torch.float64, device="cuda") for h in H]
    V = [torch.empty_like(h) for h in H]
    assert (nb.diag_batch_device(H, E, V) == 0).all()
    for i in list(range(len(H0))) + [count - 1]:
        h, e, v = H0[i % len(H0)], E[i], V[i]
        Hf, m = h + torch.triu(h, 1).T, h.shape[0]
        assert torch.linalg.norm(v @ Hf - e[:, None] * v, dim=1).max().item() <= 1e-12 * e.abs().max().item() * m ** 0.5
        assert (v @ v.T - torch.eye(m, dtype=torch.float64, device="cuda")).abs().max().item() < 1e-10


@pytest.mark.parametrize("n", [40, 96, 150, 300, 700, 1100])
def test_columns_that_are_reduced_already(nb, oracle, n):
    """Columns without a reflector: all of them (a subspace with one ancestor), whole panels, every other one."""
    i, j = np.indices((n, n))
    blocks = []
    for zero in (i != j, j > i + 1, (i < n // 2) & (j >= n // 2), (i != j) & (i < n - 20), (i % 2 == 0) & (j > i + 1),
                 (i % 48 < 32) & (j > i + 1)):
        h = np.triu(np.random.default_rng(n).standard_normal((n, n)))
        h[zero] = 0.0
        blocks.append(h)
    check_all(nb, oracle, blocks, small_max_n=96)
