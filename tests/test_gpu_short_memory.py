"""Index builds while device memory is nearly full: where the records and the table still fit but
the list of shared contexts does not, the index is built without it and joins all groups."""
import numpy as np
import pytest

import kssdgpu
import oracle

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _pairs(n, groups, seed):
    """Records of contexts held by two of n genomes each."""
    rng = np.random.default_rng(seed)
    a = rng.integers(0, n, groups)
    b = (a + rng.integers(1, n, groups)) % n
    obj = rng.integers(0, 16, (groups, 2))
    ctx = np.arange(groups, dtype=np.uint64) * np.uint64(3)
    keys = [np.sort(np.concatenate([(ctx[a == g] << np.uint64(20)) | obj[a == g, 0].astype(np.uint64),
                                    (ctx[b == g] << np.uint64(20)) | obj[b == g, 1].astype(np.uint64)]))
            for g in range(n)]
    return np.concatenate(keys), np.cumsum([0] + [len(k) for k in keys]).astype(np.uint64)


def test_index_without_its_list():
    import torch
    n = 40
    keys, offs = _pairs(n, 2_000_000, 8)
    rec = oracle.build_index(keys, offs)
    want = oracle.self_lower_all(rec, keys, offs)

    def build():
        before = kssdgpu.launch_count()
        idx = kssdgpu.Index.from_records(rec, n)
        return idx, kssdgpu.launch_count() - before

    idx, listed = build()
    got = idx.self_lower(kssdgpu.SELF_SCAN)
    np.testing.assert_array_equal(got[0], want[0])
    idx.close()
    bare = 0
    for room in range(560, 0, -24):
        kssdgpu.trim()
        torch.cuda.empty_cache()
        filler = torch.empty(torch.cuda.mem_get_info()[0] - room * MB, dtype=torch.uint8, device="cuda")
        try:
            idx, launches = build()
        except kssdgpu.KssdGpuError:  # the rest does not fit either
            break
        if launches == listed:
            idx.close()
            del filler
            continue
        bare += 1
        for flags in (kssdgpu.SELF_SCAN, 0):
            got = idx.self_lower(flags)
            np.testing.assert_array_equal(got[0], want[0])
            np.testing.assert_array_equal(got[1], want[1])
        del filler
        torch.cuda.empty_cache()
        got = idx.self_lower(kssdgpu.SELF_DENSE)  # by alleles
        np.testing.assert_array_equal(got[0], want[0])
        np.testing.assert_array_equal(got[1], want[1])
        idx.close()
    else:
        pytest.fail("every build fitted")
    del filler
    torch.cuda.empty_cache()
    assert bare >= 2
    kssdgpu.trim()
