"""Indexes built from sketches whose samples begin and end around the span of keys that a
warp takes: empty samples, several in one span, one over several spans; and keys out of
order at the ends of spans and samples."""
import numpy as np
import pytest

import kssdgpu
import oracle

pytestmark = pytest.mark.gpu

SIZES = [[1], [512], [513], [0, 0, 511, 1, 512, 0, 1024, 0], [0] * 40 + [3] + [0] * 700 + [2] + [0] * 5,
         [1] * 1030, [511, 2, 510, 0, 1, 1537, 31, 33, 4000, 0, 0]]


def sketch(sizes):
    rng = np.random.default_rng(len(sizes))
    parts = [np.sort(rng.choice(1 << 15, s, replace=False).astype(np.uint64) << np.uint64(18)) for s in sizes]
    offs = np.zeros(len(sizes) + 1, dtype=np.uint64)
    offs[1:] = np.cumsum(sizes)
    return np.concatenate(parts), offs


@pytest.mark.parametrize("sizes", SIZES, ids=lambda s: f"{len(s)}samples")
def test_sample_boundaries(sizes):
    keys, offs = sketch(sizes)
    rec = oracle.build_index(keys, offs)
    idx = kssdgpu.Index.from_sketch(kssdgpu.Sketch(keys, offs, []))
    for got, want in zip(idx.count_block(keys, offs, kssdgpu.UNIQUE),
                         oracle.count_block(rec, len(sizes), keys, offs, unique=True)):
        np.testing.assert_array_equal(got, want)
    idx.close()


@pytest.mark.parametrize("at", [1, 511, 512, 513, 1023, 1024, 1599])
def test_keys_out_of_order(at):
    keys, offs = sketch([1600, 5])
    keys[at] = keys[at - 1] - np.uint64(1)
    with pytest.raises(kssdgpu.KssdGpuError) as e:
        kssdgpu.Index.from_sketch(kssdgpu.Sketch(keys, offs, []))
    assert e.value.code == 3  # KSSDGPU_ERR_UNSORTED


@pytest.mark.parametrize("at", [1, 511, 512, 513, 1024])
def test_samples_start_low(at):
    keys, _ = sketch([1600])
    keys[at:] = keys[:1600 - at]  # the second sample starts below the first one's end
    offs = np.array([0, at, 1600], dtype=np.uint64)
    rec = oracle.build_index(keys, offs)
    idx = kssdgpu.Index.from_sketch(kssdgpu.Sketch(keys, offs, []))
    for got, want in zip(idx.count_block(keys, offs), oracle.count_block(rec, 2, keys, offs)):
        np.testing.assert_array_equal(got, want)
    idx.close()
