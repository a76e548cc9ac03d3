"""Server and no-allocation counts on indexes whose contexts are walked one by one (one species,
conflicts): requests of less than a chunk, of several, and one that fills a batch."""
import ctypes as C

import numpy as np
import pytest

import kssdgpu
import oracle
from test_gpu_wide import _species

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("unique", [False, True])
@pytest.mark.parametrize("kind", ["species", "conflicts"])
def test_walks(kind, unique):
    import torch
    n = 90
    keys, offs = _species(n, 5000, 0.8, 0.03, 20, 41)
    if kind == "conflicts":  # every seventh key with a second object
        parts = [np.unique(np.concatenate([keys[int(a):int(b)], keys[int(a):int(b):7] ^ np.uint64(1 << 6)]))
                 for a, b in zip(offs[:-1], offs[1:])]
        keys, offs = np.concatenate(parts), np.cumsum([0] + [len(p) for p in parts]).astype(np.uint64)
    rec = oracle.build_index(keys, offs)
    idx = kssdgpu.Index.from_records(rec, n)
    rng = np.random.default_rng(5)
    all_keys = np.unique(keys)
    reqs = [keys[:0], all_keys[:1], all_keys[:255], all_keys[:257], keys[int(offs[3]):int(offs[4])],
            np.sort(rng.choice(all_keys, 4097, replace=False)), all_keys]  # contexts with many objects
    qoffs = np.cumsum([0] + [len(r) for r in reqs]).astype(np.uint64)
    qkeys = np.concatenate(reqs)
    want = oracle.count_block(rec, n, qkeys, qoffs, unique=unique)
    flags = kssdgpu.UNIQUE if unique else 0
    server = kssdgpu.Server(idx, max_batch_queries=8, max_batch_keys=len(all_keys), slots=2, flags=flags)
    for _ in range(2):
        tickets = [server.submit(r) for r in reqs]
        for i, t in enumerate(tickets):
            hits, _ = server.result(t)
            got = np.zeros((4, n, 2), dtype=np.uint32)
            got[0, hits["ref"], 0], got[0, hits["ref"], 1] = hits["num_ctx"], hits["num_mut2_ctx"]
            got[1, hits["ref"], 0], got[1, hits["ref"], 1] = hits["diff_obj"], hits["diff_obj_section"]
            got[2, hits["ref"], 0], got[2, hits["ref"], 1] = hits["u_num_ctx"], hits["u_num_mut2_ctx"]
            got[3, hits["ref"], 0], got[3, hits["ref"], 1] = hits["u_diff_obj"], hits["u_diff_obj_section"]
            for g, w in zip(got, want):
                np.testing.assert_array_equal(g, w[i])
    server.close()
    dk, do = torch.from_numpy(qkeys.view(np.int64)).cuda(), torch.from_numpy(qoffs.view(np.int64)).cuda()
    out = [torch.full((len(reqs) * n,), -1, dtype=torch.int64, device="cuda") for _ in range(4 if unique else 2)]
    lib = kssdgpu.gpu_lib()
    lib.kssdgpu_count_block_noalloc.argtypes = [C.c_void_p] * 3 + [C.c_int] * 3 + [C.c_uint] + [C.c_void_p] * 5
    ptr = [o.data_ptr() for o in out] + [None] * (4 - len(out))
    torch.cuda.synchronize()
    kssdgpu._check(lib.kssdgpu_count_block_noalloc(idx.handle, dk.data_ptr(), do.data_ptr(), len(reqs), 0, 0, flags,
                                                   *ptr, None))
    idx.sync()
    for g, w in zip(out, want):
        np.testing.assert_array_equal(g.cpu().numpy().view(np.uint32).reshape(len(reqs), n, 2), w)
    idx.close()
