"""Blocks counted stripe by stripe with chunks so short and so many that a warp takes two or four of
them at a time, with queries without entries in most stripes, and one chunk more or less than the
warps' takes come to."""
import numpy as np
import pytest

import kssdgpu
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("conflict,unique", [(False, False), (False, True), (True, True)])
@pytest.mark.parametrize("nq,per", [(700, 300), (1900, 300), (1901, 40)])
def test_takes(nq, per, conflict, unique):
    rng = np.random.default_rng(nq + per)
    n = 24
    space = 400_000
    refs = []
    for _ in range(n):
        k = (np.sort(rng.choice(space, 20000, replace=False)).astype(np.uint64) << np.uint64(20)) \
            | rng.integers(0, 4, 20000).astype(np.uint64)
        refs.append(np.unique(np.concatenate([k, k[::9] ^ np.uint64(32)])) if conflict else k)
    rk, ro = np.concatenate(refs), np.cumsum([0] + [len(r) for r in refs]).astype(np.uint64)
    rec = oracle.build_index(rk, ro)
    idx = kssdgpu.Index.from_records(rec, n)
    stripes = idx.filter(2048)["stripes"]
    assert stripes >= 128
    queries = [np.sort(rng.choice(space, int(rng.integers(0, per)), replace=False).astype(np.uint64) << np.uint64(20))
               for _ in range(nq)]
    offs = np.cumsum([0] + [len(q) for q in queries]).astype(np.uint64)
    keys = np.concatenate(queries)
    want = oracle.count_block(rec, n, keys, offs, unique=unique)
    import torch
    dk, do = torch.from_numpy(keys.view(np.int64)).cuda(), torch.from_numpy(offs.view(np.int64)).cuda()
    out = [torch.full((nq * n,), -1, dtype=torch.int64, device="cuda") for _ in range(4 if unique else 2)]
    torch.cuda.synchronize()
    idx.count_block_dev(dk, do, nq, *out, flags=kssdgpu.UNIQUE if unique else 0)
    idx.sync()
    for g, w in zip(out, want):
        np.testing.assert_array_equal(g.cpu().numpy().view(np.uint32).reshape(nq, n, 2), w)
    idx.close()
