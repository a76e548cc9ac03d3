"""Chunks of blocks of few large queries (read sets), on both sides of the size from which queries count
as large and of the number of chunks that such a block gives, cut by the device and by the host."""
import ctypes as C

import numpy as np
import pytest

import kssdgpu
import oracle

pytestmark = pytest.mark.gpu

LARGE, GOAL = 32768, 5 * 148


@pytest.mark.parametrize("conflict", [False, True])
@pytest.mark.parametrize("sizes", [
    [LARGE - 1], [LARGE], [LARGE + 1, LARGE - 1], [LARGE + 1, LARGE - 2],
    [256 * GOAL - 1], [256 * GOAL], [256 * GOAL + 1],  # one chunk for each CTA, and one more
    [0, 512 * GOAL, 0, 255, 300_000],
])
def test_large_queries(sizes, conflict):
    import torch
    rng = np.random.default_rng(sum(sizes) % 9973)
    n, nq = 30, len(sizes)
    refs = [np.unique((rng.choice(1 << 18, 4000, replace=False).astype(np.uint64) << np.uint64(22))
                      | rng.integers(0, 4, 4000).astype(np.uint64)) for _ in range(n)]
    if conflict:
        refs = [np.unique(np.concatenate([r, r[::7] ^ np.uint64(16)])) for r in refs]
    rk, ro = np.concatenate(refs), np.cumsum([0] + [len(r) for r in refs]).astype(np.uint64)
    rec = oracle.build_index(rk, ro)
    idx = kssdgpu.Index.from_records(rec, n)
    queries = []
    for size in sizes:
        k = np.sort(rng.choice(1 << 20, size, replace=False).astype(np.uint64)) << np.uint64(20)
        k |= rng.integers(0, 4, size).astype(np.uint64)
        two = np.flatnonzero(rng.random(max(size - 1, 0)) < 0.02)
        k[two + 1] = k[two] + np.uint64(8)
        queries.append(np.sort(k))
    keys, offs = np.concatenate(queries), np.cumsum([0] + sizes).astype(np.uint64)
    want = oracle.count_block(rec, n, keys, offs, unique=True)
    for g, w in zip(idx.count_block(keys, offs, kssdgpu.UNIQUE), want):
        np.testing.assert_array_equal(g, w)
    dk, do = torch.from_numpy(keys.view(np.int64)).cuda(), torch.from_numpy(offs.view(np.int64)).cuda()
    out = [torch.full((nq * n,), -1, dtype=torch.int64, device="cuda") for _ in range(4)]
    lib = kssdgpu.gpu_lib()
    lib.kssdgpu_count_block_noalloc.argtypes = [C.c_void_p] * 3 + [C.c_int] * 3 + [C.c_uint] + [C.c_void_p] * 5
    ptr = [o.data_ptr() for o in out]
    for call in (lambda: idx.count_block_dev(dk, do, nq, *out, flags=kssdgpu.UNIQUE),
                 lambda: kssdgpu._check(lib.kssdgpu_count_block_noalloc(idx.handle, dk.data_ptr(), do.data_ptr(), nq, 0,
                                                                        0, kssdgpu.UNIQUE, *ptr, None))):
        for o in out:
            o.fill_(-1)
        torch.cuda.synchronize()
        call()
        torch.cuda.synchronize()
        for g, w in zip(out, want):
            np.testing.assert_array_equal(g.cpu().numpy().view(np.uint32).reshape(nq, n, 2), w)
    idx.sync()
    idx.close()
