"""Kept device memory: kssdgpu_trim and kssdgpu_index_trim give it back, the calls behind them make
it again, and a server's slots find room while the library holds blocks idle."""
import numpy as np
import pytest

import kssdgpu
import oracle
from test_gpu_wide import _species

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _large(seed):
    """An index whose arrays take some hundred megabytes."""
    rng = np.random.default_rng(seed)
    keys = np.sort(rng.integers(0, 1 << 63, 6_000_000, dtype=np.uint64))
    return kssdgpu.Index.from_sketch(kssdgpu.Sketch(keys=keys, offs=np.array([0, len(keys)], dtype=np.uint64),
                                                    names=["a"]))


def test_memory_is_given_back():
    n = 200
    keys, offs = _species(n, 3000, 0.9, 0.03, 20, 3)
    rec = oracle.build_index(keys, offs)
    want = oracle.count_block(rec, n, keys, offs)
    _large(1).close()
    kssdgpu.trim()
    start = _free()
    _large(2).close()
    assert start - _free() > 300 * MB
    kssdgpu.trim()
    assert start - _free() < 8 * MB
    idx = kssdgpu.Index.from_records(rec, n)
    for again in range(3):
        if again < 2:  # the first round loads the kernels, which stay
            idx.trim()
            kssdgpu.trim()
            built = _free()
        for g, w in zip(idx.count_block(keys, offs), want):
            np.testing.assert_array_equal(g, w)
        idx.self_lower(kssdgpu.SELF_DENSE)
        kssdgpu.trim()
        assert built - _free() > 16 * MB  # its scratch
        idx.trim()
        kssdgpu.trim()
        assert not again or built - _free() < 8 * MB
    idx.close()
    kssdgpu.trim()


def test_server_beside_idle_blocks():
    import torch
    n = 16
    keys, offs = _species(n, 500, 0.9, 0.03, 20, 4)
    rec = oracle.build_index(keys, offs)
    idx = kssdgpu.Index.from_records(rec, n)
    torch.cuda.empty_cache()
    kssdgpu.trim()
    large = _large(5)
    filler = torch.empty(_free() - 100 * MB, dtype=torch.uint8, device="cuda")
    large.close()  # its blocks stay with the library: 100 MB are free outside
    assert _free() < 120 * MB
    server = kssdgpu.Server(idx, max_batch_queries=4, max_batch_keys=25 << 20, max_hits=64, slots=1)
    want = oracle.count_block(rec, n, keys[:int(offs[1])], offs[:2])
    hits, _ = server.result(server.submit(keys[:int(offs[1])]))
    assert np.array_equal(hits["num_ctx"], want[0][0, :, 0][hits["ref"]]) and len(hits) == (want[0][0, :, 0] > 0).sum()
    server.close()
    del filler
    torch.cuda.empty_cache()
    idx.close()
    kssdgpu.trim()
