"""Context counts per reference at the reference counts where the kernel changes its way:
one and two sums of a CTA in shared memory, and none."""
import numpy as np
import pytest

import kssdgpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nref", [1, 33, 12800, 12801, 25600, 25601])
@pytest.mark.parametrize("conflict,ignore", [(False, False), (True, False), (True, True)])
def test_ref_counts(nref, conflict, ignore):
    rng = np.random.default_rng(nref)
    ctx = rng.integers(0, 3000, 9000)
    gid = np.minimum(rng.integers(0, nref, 9000), rng.integers(0, nref, 9000))
    obj = rng.integers(0, 3, 9000)
    rec = np.unique((ctx.astype(np.uint64) << np.uint64(40)) | (gid.astype(np.uint64) << np.uint64(20)) |
                    obj.astype(np.uint64))
    out = np.zeros(len(rec), dtype=kssdgpu.REC_DTYPE)
    out["ctxgid"], out["obj"] = rec >> np.uint64(20), (rec & np.uint64(0xFFFFF)).astype(np.uint32)
    idx = kssdgpu.Index.from_records(out, nref)
    got, got_unique = idx.ref_ctx_counts(conflict, ignore)
    run, size = np.unique(rec >> np.uint64(20), return_counts=True)  # (context, gid) runs
    g = (run & np.uint64(0xFFFFF)).astype(np.int64)
    keep = size if not conflict else np.where(size > 1, 0 if ignore else 1, 1)
    want = np.bincount(g, weights=keep, minlength=nref)
    owners, first, count = np.unique(run >> np.uint64(20), return_index=True, return_counts=True)
    sole = first[(count == 1) & (~np.bool_(ignore) | (size[first] == 1))]
    np.testing.assert_array_equal(got, want.astype(np.uint32))
    np.testing.assert_array_equal(got_unique, np.bincount(g[sole], minlength=nref).astype(np.uint32))
    idx.close()
