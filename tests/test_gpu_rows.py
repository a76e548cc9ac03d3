"""Lower blocks and shared-memory rows, counted an entry a lane: references around the sizes
where a row passes the shared memory that a kernel has without asking for more, queries
around a warp's and a CTA's round, with one and with many filter stripes."""
import numpy as np
import pytest

import kssdgpu
import oracle
from fixtures import samples_to_sketch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 1100, 1400, 1536, 2200, 3000, 3072, 3073])
@pytest.mark.parametrize("stripe_bytes", [0, 512])
def test_rows(n, stripe_bytes):
    rng = np.random.default_rng(n)
    ctxs = 9000
    samples = [[] for _ in range(n)]
    for c in range(ctxs):  # groups of 1 to 70 genomes, some of one species, some of any
        k = min(n, int(rng.choice([1, 1, 1, 2, 3, 7, 31, 32, 70])))
        own = rng.choice(n, k, replace=False) if c % 3 else (c * 7 + np.arange(k)) % n
        base = int(rng.integers(0, 1 << 20))
        for g in own:
            samples[int(g)].append((c * 4099, base ^ (int(rng.integers(0, 4)) << 6)))
    keys, offs = samples_to_sketch(samples)
    queries = []
    for size in (0, 1, 31, 32, 33, 511, 512, 513, 4097, 8191):
        q = [(int(x) * 4099, int(rng.integers(0, 1 << 20))) for x in rng.choice(ctxs, size, replace=False)]
        if size % 2:
            q += [(x, o ^ 5) for x, o in q[::3]]  # several objects of a context
        queries.append(q)
    qkeys, qoffs = samples_to_sketch(queries)
    rec = oracle.build_index(keys, offs)
    idx = kssdgpu.Index.from_records(rec, n)
    if stripe_bytes:
        assert idx.filter(stripe_bytes)["stripes"] > 1
    for flags in (0, kssdgpu.GLOBAL_ACC, kssdgpu.SMEM_ACC):
        want = oracle.count_block(rec, n, qkeys, qoffs, unique=True)
        for g, w in zip(idx.count_block(qkeys, qoffs, kssdgpu.UNIQUE | flags), want):
            np.testing.assert_array_equal(g, w)
        want = oracle.count_block(rec, n, qkeys, qoffs)
        for g, w in zip(idx.count_block(qkeys, qoffs, flags), want):
            np.testing.assert_array_equal(g, w)
        for off in (0, n // 2):
            want = oracle.count_lower(rec, n, off, qkeys, qoffs)
            for g, w in zip(idx.count_lower(qkeys, qoffs, off, flags), want):
                np.testing.assert_array_equal(g, w)
    idx.close()
