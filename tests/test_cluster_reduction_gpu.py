"""The shared-memory reductions at the orders where a cluster of 1, 2, 4, 8 or 16 CTAs is just full or
one too small, in batches that choose the largest clusters (few blocks) and the smallest (many),
against the oracle's dsyev; and the same block to the last bit whatever cluster it gets."""
import numpy as np
import pytest

from eigcheck import check_eig

pytestmark = pytest.mark.gpu

EDGES = [65, 164, 165, 230, 231, 323, 324, 448, 449, 600]


@pytest.fixture(scope="module")
def nb():
    import nrgljubljana_b200 as m
    m.context()
    return m


def blocks_of(sizes, seed):
    rng = np.random.default_rng(seed)
    out = []
    for k, n in enumerate(sizes):
        a = rng.standard_normal((n, n))
        h = np.triu(a + a.T)
        if k % 3 == 1:  # a column that is already reduced (tau = 0), and a decoupled half
            h[0, 2:] = 0.0
            h[: n // 2, n // 2:] = 0.0
        out.append(h)
    return out


@pytest.mark.parametrize("copies", [1, 4])
def test_cluster_edges(nb, oracle, copies):
    sizes = EDGES * copies  # one of each: the clusters grow; four: more CTAs than SMs
    blocks = blocks_of(sizes, 31 + copies)
    got = nb.diagonalisations(blocks)
    for h, g in list(zip(blocks, got))[: len(EDGES)]:
        w, v = oracle.diagonalise(h)
        check_eig(h, g.val, g.vec, w, v, oracle)


@pytest.mark.parametrize("n", [100, 301, 448])
def test_same_result_in_any_cluster(nb, n):
    blocks = blocks_of([n] * 12, 7 * n)
    together = nb.diagonalisations(blocks)
    for k in (0, 1, 11):
        alone = nb.diagonalisations([blocks[k]])[0]
        assert np.array_equal(alone.val, together[k].val) and np.array_equal(alone.vec, together[k].vec)


@pytest.mark.parametrize("scale", [1.0, 1e-140, 1e140])
def test_one_cta_solver_orders(nb, oracle, scale):
    """Every order the one-CTA solver can be given (its merge trees and tile remainders differ), with
    random, graded, degenerate and decoupled matrices, at the scale where squares nearly overflow."""
    rng = np.random.default_rng(3)
    ctx = nb.Context()
    ctx.set_tuning(small_max_n=96)
    blocks = []
    for n in range(1, 97):
        a = rng.standard_normal((n, n))
        h = np.triu(a + a.T)
        if n % 4 == 1:
            h = np.diag(np.repeat(rng.standard_normal((n + 2) // 3), 3)[:n])  # exactly degenerate
        elif n % 4 == 2:
            h = np.triu(a * 0.1, 1) + np.diag(2.0 ** (-np.arange(n) / 2.0))
        elif n % 4 == 3:
            h[: n // 2, n // 2:] = 0.0
        blocks.append(h * scale)
    got = nb.diagonalisations(blocks, ctx=ctx, check_upper=False)
    for h, g in zip(blocks, got):
        w, v = oracle.diagonalise(h)
        if scale == 1.0:
            check_eig(h, g.val, g.vec, w, v, oracle)
        else:  # check_eig's norms underflow or overflow; the scaled problem is the same one
            check_eig(h / scale, g.val / scale, g.vec, w / scale, v, oracle)


@pytest.mark.parametrize("sizes", [[601], [625, 640, 703], [768, 1025, 1300], [608] * 60 + [801]])
def test_group_reduction(nb, oracle, sizes):
    """The reduction by groups of CTAs: one block over the whole chip, several beside one another and
    beside clusters, more blocks than groups (a queue each); panel remainders, decoupled halves."""
    blocks = blocks_of(sizes + [300, 70], 5)
    got = nb.diagonalisations(blocks)
    for k in {0, 1, len(sizes) // 2, len(sizes) - 1, len(sizes)}:
        w, v = oracle.diagonalise(blocks[k])
        check_eig(blocks[k], got[k].val, got[k].vec, w, v, oracle)
