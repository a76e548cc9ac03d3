"""The count autotuner on a block of one species: it times what later calls run (wide groups on the
tensor cores), and a later call takes that route whatever the tuner chose for others."""
import numpy as np
import pytest

import kssdgpu
import oracle
from test_gpu_wide import _species

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("unique", [False, True])
def test_tuned_block_of_one_species(unique):
    import torch
    n, nq = 200, 101
    keys, offs = _species(n, 1500, 0.9, 0.03, 20, 21)
    rec = oracle.build_index(keys, offs)
    want = oracle.count_block(rec, n, keys[:int(offs[nq])], offs[:nq + 1], unique=unique)
    idx = kssdgpu.Index.from_records(rec, n)
    flags = kssdgpu.UNIQUE if unique else 0
    dk = torch.from_numpy(keys.view(np.int64)).cuda()
    do = torch.from_numpy(offs[:nq + 1].view(np.int64)).cuda()
    out = [torch.full((nq * n,), -1, dtype=torch.int64, device="cuda") for _ in range(4 if unique else 2)]

    def launches(call):
        before = kssdgpu.launch_count()
        got = call()
        torch.cuda.synchronize()
        return kssdgpu.launch_count() - before, got

    def count(f):
        return launches(lambda: idx.count_block_dev(dk, do, nq, *out, flags=flags | f))[0]

    walked, wide = count(kssdgpu.GLOBAL_ACC), count(0)
    assert wide > walked
    tuning, picked = launches(lambda: idx.count_tune(dk, do, nq, *out, flags=flags))
    # four runs a candidate: all but the shared rows (one launch each) through the tensor cores
    assert tuning >= 4 * (picked["candidates"] - 2) * wide
    assert count(0) >= wide - 2  # the filter or the chunks may have gone
    for g, w in zip(out, want):
        np.testing.assert_array_equal(g.cpu().numpy().view(np.uint32).reshape(nq, n, 2), w)
    idx.close()
