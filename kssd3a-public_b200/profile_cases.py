"""Small, self-contained launches of the hot kernels for one-kernel ncu captures.

    python kssd3a-public_b200/profile_cases.py scan    # 2,000-genome self join, 3 steps
    python kssd3a-public_b200/profile_cases.py scanbig # 5,000 small genomes: triangle beyond L2
    python kssd3a-public_b200/profile_cases.py dense   # 512-genome one-species dense join, 2 steps
    python kssd3a-public_b200/profile_cases.py rect    # 2,000 queries x 4,000 references, 4 batched counts
    python kssd3a-public_b200/profile_cases.py denseprobe  # 128 queries x 512 one-species references, 3 counts
    python kssd3a-public_b200/profile_cases.py lower   # 2,000 genomes against themselves, 3 lower counts
    python kssd3a-public_b200/profile_cases.py sketch  # 12 genomes of 4 Mbp, sketched twice
    python kssd3a-public_b200/profile_cases.py values  # matrix values of 3,000 genomes, 2 launches

Each case builds its index from a seeded synthetic sketch (the generators of the
benchmark), runs a few launches of the kernel under study on cuda:0 and exits, so
that a capture (`ncu -k <kernel> -s <skip> -c <count> ...`) holds a few GB of device
memory at most and ends by itself.  No timing is printed: times taken under a
profiler are not measurements.
"""
from __future__ import annotations

import os
import sys

import numpy as np

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
import torch  # noqa: E402

import kssdgpu  # noqa: E402

THREADS = os.cpu_count() or 8


def case_scan(dev, st):
    n = 2000
    sk = kssdgpu.synth(n_samples=n, n_clusters=n // 10, size_dist=kssdgpu.SIZE_LOGNORMAL, len_median=4e6,
                       len_sigma=0.37, len_min=1e6, len_max=12e6, sub_lo=0.001, sub_hi=0.2, seed=20261203 + 2,
                       sample_seed=20261203 + 2, threads=THREADS)
    idx = kssdgpu.Index.from_sketch(sk)
    cells = n * (n - 1) // 2
    a = torch.zeros(cells, dtype=torch.int64, device=dev)
    b = torch.zeros_like(a)
    for _ in range(3):
        idx.self_lower_dev(a, b, flags=kssdgpu.SELF_SCAN, stream=st)
    torch.cuda.synchronize()
    idx.close()


def case_scanbig(dev, st):
    """5,000 genomes of 0.5-2 Mbp: the packed triangle (12.5M cells, 200 MB) is larger than
    L2, so each touched cell's line comes from memory; about 1 GB on the device."""
    n = 5000
    sk = kssdgpu.synth(n_samples=n, n_clusters=n // 10, size_dist=kssdgpu.SIZE_LOGNORMAL, len_median=1e6,
                       len_sigma=0.37, len_min=5e5, len_max=2e6, sub_lo=0.001, sub_hi=0.2, seed=20261203 + 2,
                       sample_seed=20261203 + 2, threads=THREADS)
    idx = kssdgpu.Index.from_sketch(sk)
    cells = n * (n - 1) // 2
    a = torch.zeros(cells, dtype=torch.int64, device=dev)
    b = torch.zeros_like(a)
    for _ in range(3):
        idx.self_lower_dev(a, b, flags=kssdgpu.SELF_SCAN, stream=st)
    torch.cuda.synchronize()
    print("entries", int(sk.offs[-1]))
    idx.close()


def case_dense(dev, st):
    n = 512
    sk = kssdgpu.synth(n_samples=n, n_clusters=1, size_dist=kssdgpu.SIZE_LOGNORMAL, len_median=4e6, len_sigma=0.2,
                       len_min=2e6, len_max=8e6, sub_lo=0.001, sub_hi=0.02, seed=7, sample_seed=7, threads=THREADS)
    idx = kssdgpu.Index.from_sketch(sk)
    cells = n * (n - 1) // 2
    a = torch.zeros(cells, dtype=torch.int64, device=dev)
    b = torch.zeros_like(a)
    for _ in range(2):
        idx.self_lower_dev(a, b, flags=kssdgpu.SELF_DENSE, stream=st)
    torch.cuda.synchronize()
    print("alleles", idx.dense_alleles())
    idx.close()


def case_denseprobe(dev, st):
    """The batched probe on a one-species index: 512 references and 128 new members of the
    species (context groups of hundreds of postings, walked by whole warps)."""
    ref = kssdgpu.synth(n_samples=512, n_clusters=1, size_dist=kssdgpu.SIZE_LOGNORMAL, len_median=4e6, len_sigma=0.2,
                        len_min=2e6, len_max=8e6, sub_lo=0.001, sub_hi=0.02, seed=7, sample_seed=7, threads=THREADS)
    qry = kssdgpu.synth(n_samples=128, n_clusters=1, role=kssdgpu.ROLE_OWNLEN, size_dist=kssdgpu.SIZE_LOGNORMAL,
                        len_median=4e6, len_sigma=0.2, len_min=2e6, len_max=8e6, own_len_min=1e6, own_len_max=8e6,
                        sub_lo=0.001, sub_hi=0.02, seed=7, sample_seed=8, threads=THREADS)
    idx = kssdgpu.Index.from_sketch(ref)
    dk = torch.from_numpy(qry.keys.view(np.int64)).to(dev)
    do = torch.from_numpy(qry.offs.view(np.int64)).to(dev)
    c = torch.zeros(qry.n * ref.n, dtype=torch.int64, device=dev)
    o = torch.zeros_like(c)
    for _ in range(3):
        idx.count_block_dev(dk, do, qry.n, c, o, flags=kssdgpu.GLOBAL_ACC, stream=st)
    torch.cuda.synchronize()
    print("keys", int(qry.offs[-1]), "credits", int((c & 0xFFFFFFFF).sum().item()))
    idx.close()


def case_rect(dev, st):
    nr, nq = 4000, 2000
    ref = kssdgpu.synth(n_samples=nr, n_clusters=nr // 10, size_dist=kssdgpu.SIZE_LOGNORMAL, len_median=4e6,
                        len_sigma=0.37, len_min=1e6, len_max=12e6, sub_lo=0.001, sub_hi=0.2, seed=20261206,
                        sample_seed=20261206, threads=THREADS)
    qry = kssdgpu.synth(n_samples=nq, n_clusters=nr // 10, role=kssdgpu.ROLE_OWNLEN, size_dist=kssdgpu.SIZE_LOGNORMAL,
                        len_median=4e6, len_sigma=0.37, len_min=1e6, len_max=12e6, own_len_min=5e4,
                        own_len_max=12e6, sub_lo=0.001, sub_hi=0.2, seed=20261206, sample_seed=20261207,
                        threads=THREADS)
    idx = kssdgpu.Index.from_sketch(ref)
    dk = torch.from_numpy(qry.keys.view(np.int64)).to(dev)
    do = torch.from_numpy(qry.offs.view(np.int64)).to(dev)
    c = torch.zeros(nq * nr, dtype=torch.int64, device=dev)
    o = torch.zeros_like(c)
    for i in range(4):
        idx.count_block_dev(dk, do, nq, c, o, flags=kssdgpu.NO_ZERO if i else 0, stream=st)
    torch.cuda.synchronize()
    print("keys", int(qry.offs[-1]))
    idx.close()


def case_lower(dev, st):
    """The batched probe where every key is in the index: a lower block of all its genomes."""
    n = 2000
    sk = kssdgpu.synth(n_samples=n, n_clusters=n // 10, size_dist=kssdgpu.SIZE_LOGNORMAL, len_median=4e6,
                       len_sigma=0.37, len_min=1e6, len_max=12e6, sub_lo=0.001, sub_hi=0.2, seed=20261203 + 2,
                       sample_seed=20261203 + 2, threads=THREADS)
    idx = kssdgpu.Index.from_sketch(sk)
    dk = torch.from_numpy(sk.keys.view(np.int64)).to(dev)
    do = torch.from_numpy(sk.offs.view(np.int64)).to(dev)
    c = torch.zeros(n * n, dtype=torch.int64, device=dev)
    o = torch.zeros_like(c)
    for _ in range(3):
        idx.count_block_dev(dk, do, n, c, o, lower=True, stream=st)
    torch.cuda.synchronize()
    print("keys", int(sk.offs[-1]))
    idx.close()


def case_sketch(dev, st):
    rng = np.random.default_rng(20261203)
    genomes = [[rng.choice(np.frombuffer(b"ACGT", dtype=np.uint8), 4000000).tobytes()] for _ in range(12)]
    for _ in range(2):
        keys, _ = kssdgpu.sketch(genomes)
    print("keys", len(keys))


def case_values(dev, st):
    """3,000 genomes of species of ten, random ANI within a species, nothing shared outside."""
    n = 3000
    rng = np.random.default_rng(20261203)
    size = rng.integers(12000, 20000, n).astype(np.uint32)
    q, r = np.tril_indices(n, -1)
    own = np.flatnonzero(q // 10 == r // 10)
    ctx = (rng.uniform(0.05, 0.9, len(own)) * 12000).astype(np.uint64)
    diff = (rng.uniform(0.05, 0.9, len(own)) * ctx).astype(np.uint64)
    lc, lo = np.zeros(len(q), dtype=np.uint64), np.zeros(len(q), dtype=np.uint64)
    lc[own] = ctx | ((diff // 4) << np.uint64(32))                    # num_ctx, num_mut2_ctx
    lo[own] = diff | ((diff + diff // 3) << np.uint64(32))            # diff_obj, diff_obj_section
    up = lambda a: torch.from_numpy(a).to(dev)  # noqa: E731
    d_size, d_lc, d_lo = up(size.view(np.int32)), up(lc.view(np.int64)), up(lo.view(np.int64))
    value = torch.zeros(len(q), dtype=torch.float64, device=dev)
    listed, nlisted = torch.zeros(3 * 65536, dtype=torch.int64, device=dev), torch.zeros(1, dtype=torch.int64, device=dev)
    opt = kssdgpu.metric_opt(s=-1, zero_const=1, zero_value=0.0)
    for _ in range(2):
        kssdgpu.lower_metric_dev(opt, n, d_size, d_size, d_lc, d_lo, value, listed, 65536, nlisted, stream=st)
    torch.cuda.synchronize()
    print("cells of a species", len(own))


def main(argv):
    cases = {"scan": case_scan, "scanbig": case_scanbig, "dense": case_dense, "rect": case_rect,
             "denseprobe": case_denseprobe, "lower": case_lower,
             "sketch": case_sketch, "values": case_values}
    which = argv[1] if len(argv) > 1 else ""
    if which not in cases:
        print("usage: profile_cases.py scan|scanbig|dense|rect|denseprobe|lower|sketch|values", file=sys.stderr)
        return 64
    if not torch.cuda.is_available():
        print("profile_cases.py: needs a CUDA device", file=sys.stderr)
        return 1
    dev = torch.device("cuda", 0)
    cases[which](dev, torch.cuda.current_stream())
    print("ok")
    return 0


if __name__ == "__main__":
    sys.exit(main(sys.argv))
