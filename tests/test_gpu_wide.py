"""The wide join (Gram matrices of the genomes' distances to a context's major object, and
pair corrections) against the oracle, at the sizes where it can go wrong: genome counts
around the 16-genome padding, the 128-genome tile and the GEMM's column blocks, groups at
the width where they become wide, objects whose differences reach the cap, few and many
corrections (where the join with a row per allele takes over)."""
import numpy as np
import pytest

import kssdgpu
import oracle
from fixtures import samples_to_sketch

pytestmark = pytest.mark.gpu


def _species(n, contexts, held, minor, obj_bits, seed, alleles=0):
    """n genomes over `contexts` contexts, each held with probability `held`; a genome's
    object is the context's ancestor with every base changed at rate `minor`, or one of
    `alleles` equally frequent objects."""
    rng = np.random.default_rng(seed)
    top = (1 << obj_bits) - 1
    anc = rng.integers(0, top, size=(contexts, max(alleles, 1)), dtype=np.uint64)
    samples = []
    for _ in range(n):
        have = np.flatnonzero(rng.random(contexts) < held)
        obj = anc[have, rng.integers(0, max(alleles, 1), size=len(have))]
        for b in range(obj_bits // 2):
            hit = rng.random(len(have)) < minor
            obj = np.where(hit, obj ^ (rng.integers(1, 4, size=len(have)).astype(np.uint64) << np.uint64(2 * b)), obj)
        samples.append(list(zip((have * 7919).tolist(), obj.tolist())))
    return samples_to_sketch(samples, obj_bits=obj_bits)


@pytest.mark.parametrize("n,contexts,held,minor,obj_bits,alleles", [
    (2, 40, 0.9, 0.05, 20, 0),      # the smallest triangle
    (17, 300, 0.8, 0.02, 20, 0),    # one genome past the padding
    (128, 129, 0.7, 0.03, 20, 0),   # one tile, one context past a tile's depth
    (129, 64, 0.9, 0.02, 20, 0),
    (130, 400, 0.045, 0.05, 20, 0),  # group sizes on both sides of the wide width
    (200, 90, 0.9, 0.3, 32, 0),     # differences past the cap
    (200, 60, 1.0, 0.0, 20, 3),     # three alleles of equal frequency: most pairs corrected
    (1601, 25, 0.5, 0.02, 20, 0),   # the GEMM per block of columns, the last one narrow
])
def test_wide_join(n, contexts, held, minor, obj_bits, alleles):
    keys, offs = _species(n, contexts, held, minor, obj_bits, 100 + n, alleles)
    rec = oracle.build_index(keys, offs, obj_bits=obj_bits)
    want = oracle.self_lower_all(rec, keys, offs, obj_bits=obj_bits)
    idx = kssdgpu.Index.from_records(rec, n, obj_bits=obj_bits)
    for _ in range(2):  # the second call on scratch that the first one left
        got = idx.self_lower(kssdgpu.SELF_DENSE)
        np.testing.assert_array_equal(got[0], want[0])
        np.testing.assert_array_equal(got[1], want[1])
    shared = oracle_alleles(keys, obj_bits)
    assert idx.dense_alleles() == shared
    got = idx.self_lower()
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1], want[1])
    idx.close()


def oracle_alleles(keys, obj_bits):
    """Distinct objects of the contexts that several genomes hold."""
    ctx, count = np.unique(keys >> np.uint64(obj_bits), return_counts=True)
    pairs = np.unique(keys)
    return int(np.isin(pairs >> np.uint64(obj_bits), ctx[count >= 2]).sum())


def test_common_alleles_take_the_allele_rows():
    """Two alleles of equal frequency everywhere: nearly all pairs would be corrected, so
    the join with a row per allele runs; the counters are the scan's."""
    n = 1100
    keys, offs = _species(n, 600, 0.9, 0.0, 20, 5, alleles=2)
    rec = oracle.build_index(keys, offs)
    idx = kssdgpu.Index.from_records(rec, n)
    assert idx.self_choice()[0] == kssdgpu.PATH_DENSE
    got, want = idx.self_lower(), idx.self_lower(kssdgpu.SELF_SCAN)
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1], want[1])
    assert idx.dense_alleles() == oracle_alleles(keys, 20)
    idx.close()


@pytest.mark.parametrize("n,nq,contexts,unique", [(200, 101, 1500, False), (65, 304, 3000, True),
                                                  (129, 129, 2100, False), (16, 2000, 900, True)])
def test_wide_block(n, nq, contexts, unique):
    """A block of queries against an index of wide groups, narrow groups and contexts of one
    genome; every third query holds some contexts with several objects, one query is empty."""
    keys, offs = _species(n, contexts, 0.9, 0.03, 20, 300 + n)
    rng = np.random.default_rng(n)
    samples = []
    for i in range(n):  # contexts of few genomes beside the wide ones
        k = keys[int(offs[i]):int(offs[i + 1])]
        few = [((1 << 40) + int(c), int(o)) for c, o in zip(rng.integers(0, 60 * n, 40), rng.integers(0, 1 << 20, 40))]
        samples.append([(int(x) >> 20, int(x) & 0xFFFFF) for x in k] + list(dict(few).items()))
    keys, offs = samples_to_sketch(samples)
    queries = []
    for q in range(nq):
        s = samples[int(rng.integers(0, n))]
        pick = np.flatnonzero(rng.random(len(s)) < 0.8)
        own = [(s[j][0], s[j][1] ^ (int(rng.integers(1, 4)) << 4) if rng.random() < 0.2 else s[j][1]) for j in pick]
        if q % 3 == 0:
            own += [(c, o ^ 1) for c, o in own[:50]]
        queries.append([] if q == 5 else own)
    qkeys, qoffs = samples_to_sketch(queries)
    rec = oracle.build_index(keys, offs)
    idx = kssdgpu.Index.from_records(rec, n)
    flags = kssdgpu.UNIQUE if unique else 0
    for more in (0, kssdgpu.IGNORECONFLICT):
        want = oracle.count_block(rec, n, qkeys, qoffs, unique=unique, ignoreconflict=bool(more))
        before = kssdgpu.launch_count()
        walked = idx.count_block(qkeys, qoffs, flags | more | kssdgpu.GLOBAL_ACC)
        plain = kssdgpu.launch_count() - before
        for _ in range(2):
            before = kssdgpu.launch_count()
            got = idx.count_block(qkeys, qoffs, flags | more)
            assert kssdgpu.launch_count() - before > plain  # the wide groups went to the tensor cores
            for g, w, v in zip(got, want, walked):
                np.testing.assert_array_equal(g, w)
                np.testing.assert_array_equal(v, w)
    idx.close()
