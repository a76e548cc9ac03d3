"""The sketch scan's stretches, tiles and lists against the oracle: records that end around a
thread's and a CTA's part of the sequence, records shorter than a k-mer, every filter
strength from keeping all k-mers on, and a sequence that keeps many times the expected
number (the scan runs again with room for them)."""
import numpy as np
import pytest

import kssdgpu
import oracle

pytestmark = pytest.mark.gpu


def _check(samples, **kw):
    keys, offs = kssdgpu.sketch(samples, **kw)
    for i, recs in enumerate(samples):
        want = oracle.sketch_records(recs, **kw)
        np.testing.assert_array_equal(keys[int(offs[i]):int(offs[i + 1])], want, err_msg=f"sample {i}")


def _seq(rng, n):
    s = np.frombuffer(b"ACGT", dtype=np.uint8)[rng.integers(0, 4, n)].copy()
    for at in rng.integers(0, max(n, 1), n // 3000):
        s[at:at + int(rng.integers(1, 40))] = ord("N")
    low = rng.random(n) < 0.1
    s[low] |= 32
    return s.tobytes()


@pytest.mark.parametrize("drfold", [0, 2, 8])
@pytest.mark.parametrize("klen,coden,hclen,holen", [(32, 11, 0, 0), (31, 0, 11, 3), (9, 0, 3, 1)])
def test_edges(klen, coden, hclen, holen, drfold):
    rng = np.random.default_rng(klen + drfold)
    cuts = [1, 8, klen - 1, klen, klen + 1, 63, 64, 65, 127, 16383 - 300, 16384, 16385, 16384 + 31, 3, 0, 40000, 95]
    recs = [_seq(rng, n) for n in cuts]
    _check([recs[:3], [], recs[3:12], recs[12:], [b""]], klen=klen, coden_len=coden, hclen=hclen, holen=holen,
           drfold=drfold)


def test_more_than_expected():
    """A tandem repeat one of whose 37 k-mers is kept: six times the expected number."""
    for seed in range(400):
        unit = np.frombuffer(b"ACGT", dtype=np.uint8)[np.random.default_rng(seed).integers(0, 4, 37)].tobytes()
        if len(oracle.sketch_records([unit * 4], drfold=8)):
            break
    else:
        pytest.fail("no repeat with a kept k-mer")
    rng = np.random.default_rng(1)
    _check([[unit * 110000], [_seq(rng, 50000), unit * 100]], drfold=8)
