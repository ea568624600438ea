"""Which kernels reduce a batch: the batches of tests/test_streamed_reduction_gpu.py reach the streaming kernel,
those of tests/test_cluster_reduction_gpu.py the clusters and the groups (the plan follows a cost
model, and a change of it must not leave a kernel untested)."""
import re

import pytest

pytestmark = pytest.mark.gpu

EDGES = [65, 164, 165, 230, 231, 323, 324, 448, 449, 600]


@pytest.mark.parametrize("sizes,kernels", [
    ([225 + i % 65 for i in range(528)], {"tridiag_kernel"}),
    ([440 + i % 20 for i in range(420)], {"tridiag_kernel"}),
    ([600 + i % 41 for i in range(410)], {"tridiag_kernel"}),
    ([1700 + 7 * (i % 5) for i in range(8)] + [1601] * 330, {"tridiag_kernel"}),
    ([1500, 1400] + [601 + 3 * (i % 20) for i in range(30)] + [230 + 11 * (i % 30) for i in range(300)]
     + [20 + 5 * (i % 40) for i in range(200)],
     {"tridiag_grid_kernel", "tridiag_kernel", "tridiag_dsm_kernel<1>", "tridiag_smem_kernel"}),
    (EDGES, {"tridiag_dsm_kernel<8>", "tridiag_dsm_kernel<16>"}),
    (EDGES * 4, {"tridiag_dsm_kernel<1>", "tridiag_dsm_kernel<2>", "tridiag_dsm_kernel<4>", "tridiag_dsm_kernel<8>",
                 "tridiag_dsm_kernel<16>"}),
    ([768, 1025, 1300, 300, 70], {"tridiag_grid_kernel"}),
    ([170 + i % 3 for i in range(400)], {"tridiag_smem_kernel"})])
def test_kernels(sizes, kernels):
    import torch
    from torch.profiler import ProfilerActivity, profile

    import nrgljubljana_b200 as nb
    H = [torch.eye(n, dtype=torch.float64, device="cuda") for n in sizes]
    E = [torch.empty(n, dtype=torch.float64, device="cuda") for n in sizes]
    V = [torch.empty_like(h) for h in H]
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        assert (nb.diag_batch_device(H, E, V) == 0).all()
        torch.cuda.synchronize()
    seen = set()
    for e in prof.key_averages():
        m = re.search(r"(tridiag\w*_kernel)(<\d+>)?", e.key)
        if m:
            seen.add(m.group(1) + (m.group(2) or "" if "dsm" in m.group(1) else ""))
    if not seen:
        pytest.skip("the profiler recorded no kernels (another one may hold the device's counters)")
    assert kernels <= seen, seen
