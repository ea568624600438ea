"""Blocks in which numbers far below the block's norm matter: degenerate states coupled by next to
nothing, parts that are tiny beside the rest, against the oracle's dsyev."""
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
