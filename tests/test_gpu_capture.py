"""Self joins and blocks of one species captured into CUDA graphs: the first call of an index, a
call behind larger ones on the tensor cores, and replays after the index's scratch has moved."""
import numpy as np
import pytest

import kssdgpu
import oracle
from test_gpu_wide import _species

pytestmark = pytest.mark.gpu


def _capture(call):
    import torch
    side = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        call(side)
    return graph


def _same(got, want):
    import torch
    torch.cuda.synchronize()
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g.cpu().numpy().view(np.uint32).reshape(-1, 2), w.reshape(-1, 2))


def test_captured_calls():
    import torch
    n, nq, few = 300, 200, 30
    keys, offs = _species(n, 2000, 0.9, 0.03, 20, 77)
    rec = oracle.build_index(keys, offs)
    low = oracle.self_lower_all(rec, keys, offs)
    want = oracle.count_block(rec, n, keys[:int(offs[nq])], offs[:nq + 1])
    part = [w[:few] for w in want]
    idx = kssdgpu.Index.from_records(rec, n)
    assert idx.self_choice()[0] == kssdgpu.PATH_DENSE
    tri = [torch.full((n * (n - 1) // 2,), -1, dtype=torch.int64, device="cuda") for _ in range(2)]
    out = [torch.full((nq * n,), -1, dtype=torch.int64, device="cuda") for _ in range(2)]
    cut = [torch.full((few * n,), -1, dtype=torch.int64, device="cuda") for _ in range(2)]
    dk = torch.from_numpy(keys.view(np.int64)).cuda()
    do = torch.from_numpy(offs.view(np.int64)).cuda()
    # nothing ran on the index yet
    self_graph = _capture(lambda s: idx.self_lower_dev(*tri, stream=s))
    self_graph.replay()
    _same(tri, low)
    # a warm-up that leaves the tensor cores' scratch unmade
    idx.count_block_dev(dk, do, nq, *out, flags=kssdgpu.GLOBAL_ACC)
    block_graph = _capture(lambda s: idx.count_block_dev(dk, do, few, *cut, stream=s))
    block_graph.replay()
    _same(cut, part)
    # scratch made, then moved: the graphs hold none of it
    for a, b in ((cut, few), (out, nq)):
        idx.count_block_dev(dk, do, b, *a)
    _same(out, want)
    idx.self_lower_dev(*tri)
    again = _capture(lambda s: idx.self_lower_dev(*tri, stream=s))
    for t in tri + cut:
        t.fill_(-1)
    for graph in (self_graph, block_graph):
        graph.replay()
    _same(tri, low)
    _same(cut, part)
    again.replay()
    _same(tri, low)
    del self_graph, block_graph, again
    idx.close()
