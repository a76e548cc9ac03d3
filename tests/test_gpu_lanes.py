"""Ordinary blocks counted an entry a lane: indexes with conflicts and indexes whose shared
contexts are long, groups of 31 to 97 postings with runs of several objects at the ends of
a warp's 32, several objects of a query, with one and with many filter stripes."""
import numpy as np
import pytest

import kssdgpu
import oracle
from fixtures import samples_to_sketch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("conflict", [False, True])
@pytest.mark.parametrize("stripe_bytes", [0, 512])
def test_long_groups(conflict, stripe_bytes):
    rng = np.random.default_rng(17)
    n, ctxs = 97, 1200
    samples = [[] for _ in range(n)]
    for c in range(ctxs):
        k = int(rng.choice([1, 31, 32, 33, 63, 64, 65, 96, 97]))
        base = int(rng.integers(0, 1 << 20))
        twice = set(int(x) for x in rng.choice([0, 1, 15, 30, 31, 32, 62, 63, 64], 3)) if conflict else ()
        for j, g in enumerate(np.sort(rng.choice(n, k, replace=False))):
            o = base ^ (int(rng.integers(0, 4)) << 6)
            samples[int(g)].append((c * 4099, o))
            if j in twice:
                samples[int(g)] += [(c * 4099, o ^ x) for x in (3, 1 << 9)[:1 + c % 2]]
    keys, offs = samples_to_sketch(samples)
    queries = []
    for size in (1, 33, 512, 1100):
        q = [(int(x) * 4099, int(rng.integers(0, 1 << 20))) for x in rng.choice(ctxs, size, replace=False)]
        q += [(x, o ^ y) for x, o in q[::3] for y in range(1, 1 + size % 40)]  # up to 40 objects of a context
        queries.append(q)
    qkeys, qoffs = samples_to_sketch(queries)
    rec = oracle.build_index(keys, offs)
    idx = kssdgpu.Index.from_records(rec, n)
    if stripe_bytes:
        assert idx.filter(stripe_bytes)["stripes"] > 1
    for flags in (0, kssdgpu.GLOBAL_ACC, kssdgpu.SMEM_ACC):
        for ignore in (False, True):
            want = oracle.count_block(rec, n, qkeys, qoffs, unique=True, ignoreconflict=ignore)
            got = idx.count_block(qkeys, qoffs, kssdgpu.UNIQUE | flags | (kssdgpu.IGNORECONFLICT if ignore else 0))
            for g, w in zip(got, want):
                np.testing.assert_array_equal(g, w)
            want = oracle.count_block(rec, n, qkeys, qoffs, ignoreconflict=ignore)
            got = idx.count_block(qkeys, qoffs, flags | (kssdgpu.IGNORECONFLICT if ignore else 0))
            for g, w in zip(got, want):
                np.testing.assert_array_equal(g, w)
    idx.close()
