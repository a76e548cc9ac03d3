"""Records that end within a k-mer of the end of a thread's 128 positions and of a block's 32,768, an
empty record on the edge itself, samples that change there, and a sequence that ends there."""
import numpy as np
import pytest

import kssdgpu
import oracle

pytestmark = pytest.mark.gpu

SPAN, TILE = 128, 32768


def _seq(rng, n):
    return np.frombuffer(b"ACGTacgt", dtype=np.uint8)[rng.integers(0, 8, n)].tobytes()


@pytest.mark.parametrize("klen,coden,hclen,holen", [(32, 11, 0, 0), (31, 0, 11, 3), (9, 0, 3, 1)])
@pytest.mark.parametrize("at", range(8))
def test_edges(klen, coden, hclen, holen, at):
    rng = np.random.default_rng(klen * 100 + at)
    off = [-klen, 1 - klen, -1, 0, 1, klen - 2, klen - 1, klen][at]
    # one record end near each edge, several of them at the third tile's
    cuts = [SPAN + off, 40 * SPAN - off, TILE + off, TILE + 3 * SPAN, 2 * TILE - 1, 2 * TILE, 2 * TILE, 2 * TILE + 1,
            2 * TILE + klen - 1, 3 * TILE + off]
    if at % 2:
        cuts.append(3 * TILE + off + klen)
    cuts = sorted(cuts)
    seq = _seq(rng, cuts[-1])
    recs = [seq[a:b] for a, b in zip([0] + cuts[:-1], cuts)]
    assert [sum(map(len, recs[:i + 1])) for i in range(len(recs))] == cuts and b"" in recs
    for samples in ([recs], [recs[:3], recs[3:6], [], recs[6:7], recs[7:]]):
        for drfold in (0, 4):
            prm = dict(klen=klen, coden_len=coden, hclen=hclen, holen=holen, drfold=drfold)
            keys, offs = kssdgpu.sketch(samples, **prm)
            for i, s in enumerate(samples):
                np.testing.assert_array_equal(keys[int(offs[i]):int(offs[i + 1])], oracle.sketch_records(s, **prm))
