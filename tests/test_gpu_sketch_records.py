"""Sketches of very many short records (reads) and of records in buffers of their own, from one
thread and from several at once (the page-locked chunks serve one; the others join theirs)."""
import ctypes as C
import threading

import numpy as np
import pytest

import kssdgpu
import oracle

pytestmark = pytest.mark.gpu


def _records(samples):
    """kssdgpu_sketch_records, whatever the records' lengths."""
    recs = [r for s in samples for r in s]
    rec_offs = np.cumsum([0] + [len(r) for r in recs]).astype(np.uint64)
    samp = np.cumsum([0] + [len(s) for s in samples]).astype(np.uint64)
    offs = np.zeros(len(samples) + 1, dtype=np.uint64)
    keys = np.zeros(int(rec_offs[-1]) // 100 + 4096, dtype=np.uint64)
    prm = kssdgpu._SketchParams(32, 11, 0, 0, 8, 0)
    kssdgpu._check(kssdgpu.gpu_lib().kssdgpu_sketch_records((C.c_char_p * max(len(recs), 1))(*recs), rec_offs, len(recs),
                                                            samp, len(samples), C.byref(prm), keys.ctypes.data, len(keys),
                                                            offs))
    return keys[:int(offs[-1])], offs


def _reads(rng, n, length):
    seq = np.frombuffer(b"ACGT", dtype=np.uint8)[rng.integers(0, 4, n * length)].tobytes()
    recs = [seq[i * length:(i + 1) * length] for i in range(n)]
    return [recs[:n // 3] + [b""], [], recs[n // 3:]]


def _check(samples):
    want = [oracle.sketch_records(s) for s in samples]
    for keys, offs in (kssdgpu.sketch(samples), _records(samples)):
        for i, w in enumerate(want):
            np.testing.assert_array_equal(keys[int(offs[i]):int(offs[i + 1])], w)


@pytest.mark.parametrize("n,length", [(7, 150), (13000, 150), (15000, 150), (2000, 1000), (2100, 1000), (3, 900_000)])
def test_short_records(n, length):
    _check(_reads(np.random.default_rng(n), n, length))


def test_threads_at_once():
    failed = []

    def work(t):
        try:
            for i in range(3):
                _check(_reads(np.random.default_rng(10 * t + i), 40, 100_000))
        except BaseException as e:  # noqa: BLE001
            failed.append(e)

    team = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in team:
        t.start()
    for t in team:
        t.join()
    assert not failed, failed
