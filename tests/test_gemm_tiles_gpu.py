"""Tile edges of the batched GEMM (tiles of 32 and 64, chunks of 16 in k, copies of 8 and 16 bytes): sizes
around every edge, each orientation of both operands, operands at odd offsets and leading
dimensions, several segments per output, in calls small and large enough for either tile size,
against torch in FP64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EDGES = [1, 2, 15, 16, 17, 31, 32, 33, 63, 64, 65, 130]


@pytest.fixture(scope="module")
def nb():
    import nrgljubljana_b200 as m
    m.context()
    return m


@pytest.mark.parametrize("many", [False, True])
@pytest.mark.parametrize("transA", [False, True])
@pytest.mark.parametrize("transB", [False, True])
def test_edges(nb, transA, transB, many):
    import torch
    rng = np.random.default_rng(11)
    g = torch.Generator(device="cuda")
    g.manual_seed(7)

    def view(r, c):  # an r x c view inside a NaN-filled buffer, at a random parity of offset and stride
        ld = c + int(rng.integers(0, 3))
        off = int(rng.integers(0, 3))
        buf = torch.full((off + r * ld + 2,), float("nan"), dtype=torch.float64, device="cuda")
        v = buf[off:off + r * ld].view(r, ld)[:, :c]
        v.copy_(torch.randn((r, c), generator=g, dtype=torch.float64, device="cuda"))
        return v

    terms, checks = [], []
    # 130 outputs of up to 9 tiles of 64: with the second set the call has more than 592 of them
    for rep in range(8 if many else 1):
        for q in range(60 if many else 40):
            M, N = (int(x) for x in rng.choice(EDGES, 2))
            if many and q % 3 == 0:
                M = N = 130
            C = view(M, N)
            ref = C.clone()
            for _ in range(int(rng.integers(1, 3))):
                K = int(rng.choice(EDGES))
                A, B = view(*((K, M) if transA else (M, K))), view(*((N, K) if transB else (K, N)))
                f = float(rng.choice([1.0, -0.75]))
                terms.append(nb.gemm3(C, f, A, None, B, transA=transA, transB=transB))
                ref += f * ((A.T if transA else A) @ (B.T if transB else B))
                checks.append((C, ref, A, B))
    nb.gemm3_batch(terms, host=False)
    torch.cuda.synchronize()
    for C, ref, _, _ in checks:
        # up to 2 x 130 products of unit normals per element: sums to 2^-53 x 260 x |terms| ~ 1e-13
        assert float((C - ref).abs().max()) <= 1e-12
