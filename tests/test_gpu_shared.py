"""The self join over the index's list of shared contexts against the oracle, at the sizes
where its blocks can go wrong: the last pair of a block, groups across its end, groups of 32
and 33 genomes, blocks of more genomes than they number, objects that just fit beside a
number and that do not, wide groups among the small and among the large."""
import numpy as np
import pytest

import kssdgpu
import oracle
from fixtures import samples_to_sketch

pytestmark = pytest.mark.gpu


def _groups(n, sizes, obj_bits, seed, span=None):
    """A sketch of n genomes with one context per entry of sizes, held by that many genomes
    (of a window of `span` genomes, or any), objects a few bases apart."""
    rng = np.random.default_rng(seed)
    samples = [[] for _ in range(n)]
    top = (1 << obj_bits) - 1
    for c, k in enumerate(sizes):
        lo = 0 if not span else int(rng.integers(0, n - span + 1))
        own = lo + rng.choice(span or n, size=k, replace=False)
        base = int(rng.integers(0, top, endpoint=True, dtype=np.uint64))
        for g in own:
            o = base
            for _ in range(int(rng.integers(0, 4))):
                o ^= int(rng.integers(1, 4)) << (2 * int(rng.integers(0, obj_bits // 2)))
            samples[g].append((c * 1000003, o))
    for g in range(n):  # contexts of one genome between them
        samples[g] += [(c * 1000003 + 500 + g, 1) for c in range(g % 3)]
    return samples_to_sketch(samples, obj_bits=obj_bits)


CASES = [
    (40, [2] * 2047, 20, None),            # one pair short of a block
    (40, [2] * 2048, 20, None),
    (40, [2] * 2049, 20, 10),
    (40, [32] * 9, 20, None),              # groups of 496 pairs: one starts in the block's last pairs
    (40, [32, 33] * 7 + [2], 20, None),
    (900, [2, 3, 5] * 700, 20, 30),        # blocks of up to 64 genomes, and more
    (900, [2, 3, 5] * 700, 20, None),      # hundreds of genomes: not numbered
    (70, [2, 9, 31] * 60, 26, None),       # 70 genomes a block, objects at the packed width
    (50, [2, 9, 31] * 60, 28, None),       # objects wider than that
    (50, [2, 9, 31] * 60, 32, 40),
    (820, [34, 33, 32, 3] * 40, 20, 60),   # wide from 34
    (1000, [45, 40, 34, 32, 3] * 30, 20, None),  # wide from 41: large narrow groups
]


@pytest.mark.parametrize("n,sizes,obj_bits,span", CASES, ids=[f"{c[0]}x{len(c[1])}b{c[2]}" for c in CASES])
def test_shared_list(n, sizes, obj_bits, span):
    keys, offs = _groups(n, sizes, obj_bits, 7 * n + len(sizes), span)
    rec = oracle.build_index(keys, offs, obj_bits=obj_bits)
    want = oracle.self_lower_all(rec, keys, offs, obj_bits=obj_bits)
    idx = kssdgpu.Index.from_records(rec, n, obj_bits=obj_bits)
    k = np.array(sizes)
    assert idx.self_plan_info() == dict(groups=len(k), postings=int(k.sum()), pairs=int((k * (k - 1) // 2).sum()))
    for flags in (kssdgpu.SELF_SCAN, kssdgpu.SELF_DENSE, 0, kssdgpu.SELF_SCAN):
        got = idx.self_lower(flags)
        np.testing.assert_array_equal(got[0], want[0])
        np.testing.assert_array_equal(got[1], want[1])
    idx.close()
