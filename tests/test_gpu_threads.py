"""Several threads, each with an index of its own size: the kernels with dynamic shared memory
run side by side with different amounts of it, and none finds its limit lowered by another."""
import ctypes as C
import threading

import numpy as np
import pytest

import kssdgpu
import oracle
from test_gpu_wide import _species

pytestmark = pytest.mark.gpu

ROUNDS = 40


def _values(idx, count, opt):
    cells = idx.nref * (idx.nref - 1) // 2
    out = np.zeros(cells)
    re = np.zeros(cells, dtype=kssdgpu.RECHECK_DTYPE)
    nre = C.c_uint64()
    kssdgpu._check(kssdgpu.gpu_lib().kssdgpu_self_lower_metric(idx.handle, 0, C.byref(opt), count, count,
                                                               out.ctypes.data, re.ctypes.data, cells, C.byref(nre)))
    return out


def test_threads_with_different_sizes():
    sizes = [20, 300, 900, 1500]
    start, failed = threading.Barrier(len(sizes)), []

    def work(t, n):
        try:
            keys, offs = _species(n, 40, 0.7, 0.05, 20, n)
            rec = oracle.build_index(keys, offs)
            low = oracle.self_lower_all(rec, keys, offs)
            count = np.diff(offs).astype(np.uint32)
            nq = 8
            qk, qo = keys[:int(offs[nq])], offs[:nq + 1]
            want = oracle.count_block(rec, n, qk, qo)
            idx = kssdgpu.Index.from_records(rec, n)
            # another metric a thread: with the trees, without them, raw
            opt = kssdgpu.metric_opt(**[dict(s=-1), dict(s=4), dict(s=2, raw_output=1), dict(s=1)][t])
            start.wait()
            values = None
            for i in range(ROUNDS):
                np.testing.assert_array_equal(idx.ref_ctx_counts(False, False)[0], count)
                got = idx.count_block(qk, qo, kssdgpu.SMEM_ACC)
                np.testing.assert_array_equal(got[0], want[0])
                got = idx.count_block(qk, qo)
                np.testing.assert_array_equal(got[1], want[1])
                got = idx.self_lower(kssdgpu.SELF_DENSE)
                np.testing.assert_array_equal(got[0], low[0])
                np.testing.assert_array_equal(got[1], low[1])
                v = _values(idx, count, opt)
                if i:
                    np.testing.assert_array_equal(v, values)
                values = v
            idx.close()
        except BaseException as e:  # noqa: BLE001
            start.abort()
            failed.append(e)

    team = [threading.Thread(target=work, args=(t, n)) for t, n in enumerate(sizes)]
    for t in team:
        t.start()
    for t in team:
        t.join()
    assert not failed, failed
