"""A caller's reset of the device: kssdgpu_init, and everything works in the new context; nothing
that the library kept (device blocks, page-locked chunks, the calibration model) is used again,
and an index of the old context may be closed at any time.  In a process of its own, whose
context the reset ends."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import ctypes as C, os, sys
import numpy as np
root = sys.argv[1]
for d in ("kssd3a-public_b200", "oracle"):
    sys.path.insert(0, os.path.join(root, d))
import kssdgpu, oracle

rng = np.random.default_rng(11)
n = 12
base = np.sort(rng.choice(1 << 40, 60000, replace=False).astype(np.uint64)) << np.uint64(20)
samples = [base[rng.random(len(base)) < 0.8] | rng.integers(0, 4, 1, dtype=np.uint64) for _ in range(n)]
sk = kssdgpu.Sketch(keys=np.concatenate(samples), offs=np.cumsum([0] + [len(s) for s in samples]).astype(np.uint64),
                    names=[""] * n)
assert sk.keys.nbytes > 2 << 20  # copies go through the page-locked chunks
want = oracle.build_index(sk.keys, sk.offs)
low = oracle.self_lower_all(want, sk.keys, sk.offs)
opt = kssdgpu.metric_opt(s=-1)
count = np.diff(sk.offs).astype(np.uint32)
seq = [[np.frombuffer(b"ACGT", dtype=np.uint8)[rng.integers(0, 4, 3 << 20)].tobytes()]]
sketched = oracle.sketch_records(seq[0])


def values(idx):
    out = np.zeros(n * (n - 1) // 2)
    re = np.zeros(len(out), dtype=kssdgpu.RECHECK_DTYPE)
    nre = C.c_uint64()
    kssdgpu._check(kssdgpu.gpu_lib().kssdgpu_self_lower_metric(idx.handle, 0, C.byref(opt), count, count,
                                                               out.ctypes.data, re.ctypes.data, len(re), C.byref(nre)))
    return out


def check(idx):
    assert idx.export()[0].tobytes() == want.tobytes()
    for g, w in zip(idx.self_lower(), low):
        np.testing.assert_array_equal(g, w)
    np.testing.assert_array_equal(kssdgpu.sketch(seq)[0], sketched)
    return values(idx)


first = kssdgpu.Index.from_sketch(sk)
before = check(first)
first.close()  # its blocks are kept
old = kssdgpu.Index.from_sketch(sk)
older = kssdgpu.Index.from_sketch(sk)
cuda = C.CDLL("libcuda.so.1")
for again in range(2):
    assert cuda.cuDevicePrimaryCtxReset_v2(0) == 0
    kssdgpu._check(kssdgpu.gpu_lib().kssdgpu_init(0))
    if again:
        older.close()
    idx = kssdgpu.Index.from_sketch(sk)
    np.testing.assert_array_equal(check(idx), before)
    if not again:
        old.close()  # of the old context: leaves the new one's blocks alone
    more = kssdgpu.Index.from_sketch(sk)
    np.testing.assert_array_equal(check(idx), before)
    np.testing.assert_array_equal(check(more), before)
    more.close()
    idx.close()
print("ok")
"""


def test_reset(tmp_path):
    run = subprocess.run([sys.executable, "-c", CHILD, ROOT], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0 and run.stdout.strip() == "ok", run.stdout + run.stderr
