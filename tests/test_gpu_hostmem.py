"""Host buffers of sizes around the staged copies' chunks, and device blocks handed from one
index to the next, from one and from several threads."""
import threading

import numpy as np
import pytest

import kssdgpu
import oracle

pytestmark = pytest.mark.gpu

CHUNK = 1 << 17  # keys of one staged chunk (1 MB)


def _sketch(n, seed):
    rng = np.random.default_rng(seed)
    keys = [np.unique(rng.integers(0, 1 << 64, m, dtype=np.uint64)) for m in (n // 3, n - n // 3)]
    offs = np.cumsum([0] + [len(k) for k in keys]).astype(np.uint64)
    return kssdgpu.Sketch(keys=np.concatenate(keys), offs=offs, names=["a", "b"])


def _check(n, seed):
    sk = _sketch(n, seed)
    want = oracle.build_index(sk.keys, sk.offs)
    idx = kssdgpu.Index.from_sketch(sk)
    got, _ = idx.export()
    assert got.tobytes() == want.tobytes()
    again = kssdgpu.Index.from_records(want, 2)
    assert again.export()[0].tobytes() == want.tobytes()
    idx.close()
    again.close()


@pytest.mark.parametrize("n", [1, 1000, 2 * CHUNK - 1, 2 * CHUNK, 2 * CHUNK + 1, 5 * CHUNK - 3, 33 * CHUNK + 77])
def test_staged_copies_and_kept_blocks(n):
    for seed in (n, n + 1):  # the second build takes the first one's blocks
        _check(n, seed)


def test_threads_share_the_blocks():
    failed = []

    def work(t):
        try:
            for i in range(4):
                _check(3 * CHUNK + 1000 * t + i, 10 * t + i)
        except BaseException as e:  # noqa: BLE001
            failed.append(e)

    team = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in team:
        t.start()
    for t in team:
        t.join()
    assert not failed, failed


@pytest.mark.parametrize("size", [40, (2 << 20) - 1, (2 << 20) + 5, (5 << 20) + 3])
def test_records_from_their_own_buffers(size):
    """Records as bytes (gathered from where they are) and as bytearrays (joined first)."""
    rng = np.random.default_rng(size)
    seq = np.frombuffer(b"ACGTacgtN", dtype=np.uint8)[rng.integers(0, 9, size) * (rng.random(size) < 0.999)].tobytes()
    cuts = [0, 0, *sorted(rng.integers(0, size + 1, 40).tolist()), size, size]
    recs = [seq[a:b] for a, b in zip(cuts, cuts[1:])]
    samples = [recs[:7], [], recs[7:]]
    a = kssdgpu.sketch(samples)
    b = kssdgpu.sketch([[bytearray(r) for r in s] for s in samples])
    np.testing.assert_array_equal(a[0], b[0])
    np.testing.assert_array_equal(a[1], b[1])
