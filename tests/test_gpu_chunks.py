"""Chunks of a block in global rows, at the sizes where a block gives just as many as it should and
one entry more or less, cut by the device (blocks, the no-allocation count) and by the host."""
import ctypes as C

import numpy as np
import pytest

import kssdgpu
import oracle

pytestmark = pytest.mark.gpu

GOAL = 32 * 148  # chunks that a block should give; each a multiple of 256 entries


def _block(total, nq, rng):
    """total entries in nq queries of very different sizes, every fourth from the index's contexts,
    some contexts with two objects."""
    cut = np.sort(rng.integers(0, total + 1, nq - 1))
    offs = np.concatenate([[0], cut, [total]]).astype(np.uint64)
    keys = []
    for a, b in zip(offs[:-1].astype(int), offs[1:].astype(int)):
        ctx = np.sort(rng.choice(1 << 20, b - a, replace=False).astype(np.uint64))
        k = (ctx << np.uint64(20)) | rng.integers(0, 4, b - a).astype(np.uint64)
        two = np.flatnonzero(rng.random(max(b - a - 1, 0)) < 0.02)
        k[two + 1] = k[two] + np.uint64(8)
        keys.append(np.sort(k))
    return np.concatenate(keys), offs


@pytest.mark.parametrize("conflict", [False, True])
@pytest.mark.parametrize("total", [1, 255, 257, 256 * GOAL - 1, 256 * GOAL, 256 * GOAL + 1, 512 * GOAL + 77])
def test_chunks(total, conflict):
    import torch
    rng = np.random.default_rng(total % 9973)
    n = 30
    refs = [np.unique((rng.choice(1 << 18, 4000, replace=False).astype(np.uint64) << np.uint64(22))
                      | rng.integers(0, 4, 4000).astype(np.uint64)) for _ in range(n)]
    if conflict:
        refs = [np.unique(np.concatenate([r, r[::7] ^ np.uint64(16)])) for r in refs]
    rk, ro = np.concatenate(refs), np.cumsum([0] + [len(r) for r in refs]).astype(np.uint64)
    rec = oracle.build_index(rk, ro)
    idx = kssdgpu.Index.from_records(rec, n)
    nq = 1 if total < 300 else 9
    keys, offs = _block(total, nq, rng)
    want = oracle.count_block(rec, n, keys, offs, unique=True)
    for g, w in zip(idx.count_block(keys, offs, kssdgpu.UNIQUE | kssdgpu.GLOBAL_ACC), want):
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
