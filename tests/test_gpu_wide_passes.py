"""The wide joins over more wide groups than one pass takes (131,072): one group in the last pass,
and a last pass of about 9,000; the self join, and a block with runs of several objects."""
import numpy as np
import pytest

import kssdgpu
import oracle

pytestmark = pytest.mark.gpu

PASS = 131072


def _species(n, contexts, seed):
    """n genomes; every context is held by genome 0, most by most others (so each is shared), the
    objects changed at 3 % of their bases."""
    rng = np.random.default_rng(seed)
    anc = rng.integers(0, 1 << 20, contexts, dtype=np.uint64)
    ctx = np.arange(contexts, dtype=np.uint64) * np.uint64(7919)
    out = []
    for g in range(n):
        have = np.ones(contexts, bool) if g < 2 else rng.random(contexts) < 0.9
        obj = anc[have]
        for b in range(10):
            hit = rng.random(len(obj)) < 0.03
            obj = np.where(hit, obj ^ (rng.integers(1, 4, len(obj)).astype(np.uint64) << np.uint64(2 * b)), obj)
        out.append((ctx[have] << np.uint64(20)) | obj)
    return out


def _join(parts):
    return np.concatenate(parts), np.cumsum([0] + [len(p) for p in parts]).astype(np.uint64)


def _launches(call):
    before = kssdgpu.launch_count()
    out = call()
    return out, kssdgpu.launch_count() - before


@pytest.mark.parametrize("n", [16, 17])
def test_passes(n):
    one = None  # launches of the joins with one pass
    for contexts in (PASS, PASS + 1, 140_000):
        genomes = _species(n, contexts, contexts + n)
        keys, offs = _join(genomes)
        rec = oracle.build_index(keys, offs)
        idx = kssdgpu.Index.from_records(rec, n)
        want = oracle.self_lower_all(rec, keys, offs)
        for _ in range(2):  # the second call on scratch that the first one left
            got, self_launches = _launches(lambda: idx.self_lower(kssdgpu.SELF_DENSE))
            np.testing.assert_array_equal(got[0], want[0])
            np.testing.assert_array_equal(got[1], want[1])

        rng = np.random.default_rng(n)
        queries = []
        for q in range(150):
            own = genomes[int(rng.integers(0, n))]
            own = own[rng.random(len(own)) < 0.3]
            own = np.where(rng.random(len(own)) < 0.2, own ^ np.uint64(16), own)
            if q % 3 == 0:  # contexts with two objects, up to the last ones
                own = np.concatenate([own, own[::11] ^ np.uint64(1), own[-3:] ^ np.uint64(3)])
            queries.append(np.unique(own) if q != 7 else own[:0])
        qkeys, qoffs = _join(queries)
        want = oracle.count_block(rec, n, qkeys, qoffs, unique=True)
        for _ in range(2):
            got, block_launches = _launches(lambda: idx.count_block(qkeys, qoffs, kssdgpu.UNIQUE))
            for g, w in zip(got, want):
                np.testing.assert_array_equal(g, w)
        idx.close()
        if one is None:
            one = self_launches, block_launches
        else:  # rows, products and counters once more
            assert (self_launches - one[0], block_launches - one[1]) == (3, 3)
