"""The self join of indexes whose shared contexts are all held by 33 genomes or more (no small
groups: the join of the small ones is not launched), called directly and replayed from a CUDA
graph over counters that hold other values."""
import numpy as np
import pytest

import kssdgpu
import oracle
from test_gpu_shared import _groups

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,sizes", [
    (33, [33] * 5),                  # all wide
    (40, [40, 33, 36] * 50),
    (1000, [33, 40, 35] * 20),       # all narrow: wide from 41
    (1000, [33, 41, 60] * 20),
])
def test_only_large_groups(n, sizes):
    import torch
    keys, offs = _groups(n, sizes, 20, n + len(sizes))
    rec = oracle.build_index(keys, offs)
    want = oracle.self_lower_all(rec, keys, offs)
    idx = kssdgpu.Index.from_records(rec, n)
    before = kssdgpu.launch_count()
    got = idx.self_lower(kssdgpu.SELF_SCAN)
    narrow = any(k < 41 for k in sizes) if n == 1000 else False
    wide = any(k >= 41 for k in sizes) if n == 1000 else True
    assert kssdgpu.launch_count() - before == 1 + narrow + wide  # the fill, the large groups
    for flags in (0, kssdgpu.SELF_DENSE, kssdgpu.SELF_SCAN):
        np.testing.assert_array_equal(got[0], want[0])
        np.testing.assert_array_equal(got[1], want[1])
        got = idx.self_lower(flags)
    np.testing.assert_array_equal(got[0], want[0])
    ctx = torch.zeros(n * (n - 1) // 2, dtype=torch.int64, device="cuda")
    obj = torch.zeros_like(ctx)
    side = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        idx.self_lower_dev(ctx, obj, flags=kssdgpu.SELF_SCAN, stream=side)
    for _ in range(3):
        ctx.fill_(-1)
        obj.fill_(-1)
        graph.replay()
        torch.cuda.synchronize()
        np.testing.assert_array_equal(ctx.cpu().numpy().view(np.uint32).reshape(-1, 2), want[0].reshape(-1, 2))
        np.testing.assert_array_equal(obj.cpu().numpy().view(np.uint32).reshape(-1, 2), want[1].reshape(-1, 2))
    del graph
    idx.close()
