"""The counting kernels' queues and per-warp counters against the oracle: queries of sizes
around a round, a batch and a chunk, few and many of whose contexts the index holds, more
references than a warp has cells, runs of several objects across the ends of chunks, with
one and with many filter stripes, in every accumulator mode."""
import numpy as np
import pytest

import kssdgpu
import oracle
from fixtures import samples_to_sketch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("held", [0.05, 0.6, 1.0])
@pytest.mark.parametrize("stripe_bytes", [0, 512])
def test_query_sizes(held, stripe_bytes):
    rng = np.random.default_rng(int(held * 100))
    n, ctxs = 300, 9000
    samples = [[] for _ in range(n)]
    for c in range(ctxs):  # groups of 1 to 40 genomes, some of one species, some of any
        k = int(rng.choice([1, 1, 1, 2, 3, 7, 11, 31, 32, 40]))
        own = rng.choice(n, k, replace=False) if c % 3 else (c * 7 + np.arange(k)) % n
        base = int(rng.integers(0, 1 << 20))
        for g in own:
            samples[int(g)].append((c * 4099, base ^ (int(rng.integers(0, 4)) << 6)))
    keys, offs = samples_to_sketch(samples)
    queries = []
    for size in (0, 1, 31, 32, 33, 63, 64, 65, 255, 256, 257, 511, 4095, 4096, 4097, 8191):
        c = rng.choice(ctxs, size, replace=False) * 4099
        c = np.where(rng.random(size) < held, c, c + 1 + rng.integers(0, 4000, size))
        q = [(int(x), int(rng.integers(0, 1 << 20))) for x in c]
        if size % 2:
            q += [(x, o ^ 5) for x, o in q[::3]]  # several objects of a context
        queries.append(q)
    qkeys, qoffs = samples_to_sketch(queries)
    rec = oracle.build_index(keys, offs)
    idx = kssdgpu.Index.from_records(rec, n)
    if stripe_bytes:
        assert idx.filter(stripe_bytes)["stripes"] > 1
    want = oracle.count_block(rec, n, qkeys, qoffs, unique=True)
    for flags in (0, kssdgpu.GLOBAL_ACC, kssdgpu.SMEM_ACC):
        for g, w in zip(idx.count_block(qkeys, qoffs, kssdgpu.UNIQUE | flags), want):
            np.testing.assert_array_equal(g, w)
    for off in (0, 150):
        want = oracle.count_lower(rec, n, off, qkeys, qoffs)
        for g, w in zip(idx.count_lower(qkeys, qoffs, off), want):
            np.testing.assert_array_equal(g, w)
    idx.close()
