"""The work a user of this framework has it do, as cases to be timed.

Every case is a dict of plain values; "kind" says which public entry point it goes
through:

  self     Index.self_lower_dev: the whole lower triangle of a resident index (the
           counting behind `kssd3a ani --format matrix|triangle` and `kssd3a matrix`)
  matrix   Index.from_sketch + ref_ctx_counts + self_lower on host buffers: one
           self-matrix run from a sketch in host memory, index build included
  block    Index.count_block_dev: a block of query sketches against a resident index
  detail   Index.count_detail on host buffers: the detail (TSV) run, unique contexts and
           candidate filter included
  serve    Server.submit / Server.result: requests to the serving loop
  sketch   sketch: FASTA records in host memory to sketch keys
  values   lower_metric_dev: the FP64 matrix values of a triangle of counters

Inputs are synthetic sketches in the model of the host library's generator (44-bit
contexts, 20-bit objects, one key per 256 bp, clusters of genomes derived from one
ancestor by substitutions; read sets with coverage and errors), made on the GPU by
torch because ten thousand genomes take it a fraction of a second.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kssd3a-public_b200"))
import kssdgpu  # noqa: E402

DEV = torch.device("cuda", 0)
OBJ_BITS, CTX_BITS, CODENS = 20, 44, 11
PER_BP = 1.0 / 256.0  # sketch keys per base pair at the default down-sampling
SIGN = -(1 << 63)


def listed():
    return [
        # The headline: an ANI matrix of 2,000 bacterial genomes (200 species of 10), the
        # index resident, as a service or notebook that keeps one index asks for it.
        dict(name="self-2k", kind="self", genomes=2000, per_cluster=10, bp=4e6, sub_hi=0.2),
        # The same for a large collection: the triangle (288 MB of counters) outgrows L2.
        dict(name="self-6k", kind="self", genomes=6000, per_cluster=10, bp=4e6, sub_hi=0.2),
        # A population study: 1,024 isolates of one species, most contexts shared by most genomes.
        dict(name="self-species-1k", kind="self", genomes=1024, per_cluster=1024, bp=4e6, sub_hi=0.02),
        # The smallest run: 64 genomes of 1 Mbp, sketch in host memory to matrix on the host.
        dict(name="matrix-64", kind="matrix", genomes=64, per_cluster=8, bp=1e6, sub_hi=0.05),
        # An ordinary run of the same command on 701 genomes.
        dict(name="matrix-701", kind="matrix", genomes=701, per_cluster=10, bp=4e6, sub_hi=0.2),
        # A batch of new assemblies, fragments of 50 kbp to whole genomes of 12 Mbp, against
        # a resident reference set.
        dict(name="block-1500x2k", kind="block", queries=1500, reads=False, unique=False, genomes=2000,
             per_cluster=10, bp=4e6, sub_hi=0.2),
        # Metagenomic read sets (contexts with several objects) with unique-context counting.
        dict(name="reads-40x2k", kind="block", queries=40, reads=True, unique=True, genomes=2000, per_cluster=10,
             bp=4e6, sub_hi=0.2),
        # New isolates against the index of their own species: postings lists of hundreds.
        dict(name="block-species-200x1k", kind="block", queries=200, reads=False, unique=False, genomes=1024,
             per_cluster=1024, bp=4e6, sub_hi=0.02),
        # The detail report of 333 assemblies, host buffers in, candidates out.
        dict(name="detail-333x2k", kind="detail", queries=333, genomes=2000, per_cluster=10, bp=4e6, sub_hi=0.2),
        # One request to an idle server: the latency a single caller sees.
        dict(name="serve-1x2k", kind="serve", queries=1, genomes=2000, per_cluster=10, bp=4e6, sub_hi=0.2),
        # Twelve genomes of 4 Mbp in contigs, FASTA bytes to keys.
        dict(name="sketch-12", kind="sketch", samples=12, bp=4000003, contigs=37),
        # The printed ANI values of a 3,000-genome matrix from its counters.
        dict(name="values-3k", kind="values", genomes=3000, per_cluster=10, bp=4e6, sub_hi=0.2),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above: any number of genomes, queries and samples up to
    the listed ones', clusters of any size up to one species, 1 to 6 Mbp."""
    kind = rng.choice(["self", "self", "matrix", "block", "block", "detail", "serve", "sketch", "values"])
    bp = float(rng.randrange(10, 61)) * 1e5
    if kind == "sketch":
        return dict(kind=kind, samples=_log(rng, 1, 20), bp=_log(rng, 50_000, 4_000_000), contigs=_log(rng, 1, 300))
    species = rng.random() < 0.25
    sub_hi = rng.choice([0.01, 0.02, 0.05]) if species else rng.choice([0.05, 0.1, 0.2])
    if species and kind in ("self", "block"):
        n = _log(rng, 24, 1000)
        per = n
    else:
        n = _log(rng, 24, {"self": 5000, "matrix": 800, "values": 3000}.get(kind, 2000))
        per = rng.choice([3, 5, 10, 24])
    c = dict(kind=kind, genomes=n, per_cluster=per, bp=min(bp, 4e6) if n > 700 else bp, sub_hi=sub_hi)
    if kind == "block":
        c["reads"] = rng.random() < 0.3
        c["unique"] = bool(rng.randrange(2))
        c["queries"] = _log(rng, 1, 40 if c["reads"] else 200 if species else 1500)
    elif kind == "detail":
        c["queries"] = _log(rng, 1, 333)
    elif kind == "serve":
        c["queries"] = _log(rng, 1, 48)
    return c


# ------------------------------------------------------------------ synthetic sketches


def _lengths(g, n, median, sigma):
    """Genome lengths, lognormal between a quarter of the median and three times it."""
    z = torch.randn(n, generator=g, device=DEV, dtype=torch.float64)
    return (median * torch.exp(sigma * z)).clamp(median / 4, median * 3)


def _keys(g, n):
    """Random 64-bit keys (44-bit context, 20-bit object), any bit pattern below all ones."""
    hi = torch.randint(0, (1 << 32) - 2, (n,), generator=g, device=DEV)
    lo = torch.randint(0, 1 << 32, (n,), generator=g, device=DEV)
    return (hi << 32) | lo


class _Ancestors:
    def __init__(self, g, clusters, case):
        sigma = 0.2 if clusters == 1 else 0.37
        self.count = (_lengths(g, clusters, case["bp"], sigma) * PER_BP).round().long()
        self.first = torch.cumsum(self.count, 0) - self.count
        self.keys = _keys(g, int(self.count.sum()))


def _expand(first, count):
    """Concatenated ranges [first[i], first[i] + count[i]): (owner, position) of each entry."""
    owner = torch.repeat_interleave(torch.arange(len(count), device=DEV), count)
    pos = torch.arange(len(owner), device=DEV) - (torch.cumsum(count, 0) - count)[owner]
    return owner, first[owner] + pos


def _mutate(g, keys, owner, p):
    """Each of the object's 10 bases changes with its owner's rate p."""
    for b in range(OBJ_BITS // 2):
        hit = torch.rand(len(keys), generator=g, device=DEV) < p[owner]
        sub = torch.randint(1, 4, (len(keys),), generator=g, device=DEV, dtype=torch.int64)
        keys = torch.where(hit, keys ^ (sub << (2 * b)), keys)
    return keys


def _members(g, anc, cluster, sub_hi, frac=None):
    """Keys of samples derived from their clusters' ancestors (unsorted), with their owners."""
    n = len(cluster)
    p = 0.001 + (sub_hi - 0.001) * torch.rand(n, generator=g, device=DEV)
    keep = (1 - p) ** (CTX_BITS // 2) * (1 - 0.001) ** 32
    owner, at = _expand(anc.first[cluster], anc.count[cluster])
    if frac is not None:
        part = torch.rand(len(owner), generator=g, device=DEV) < frac[owner]
        owner, at = owner[part], at[part]
    kept = torch.rand(len(owner), generator=g, device=DEV) < keep[owner]
    keys = torch.where(kept, anc.keys[at], _keys(g, len(owner)))
    return torch.where(kept, _mutate(g, keys, owner, p), keys), owner


def _finish(keys, owner, n, conflict):
    """Each sample's keys ascending as unsigned words; one object per context, or (read
    sets) no key twice.  Returns device keys (int64 bits) and offsets."""
    keys, order = torch.sort(keys ^ SIGN, stable=True)
    owner, order = torch.sort(owner[order], stable=True)
    keys = keys[order] ^ SIGN
    same = (keys[1:] ^ keys[:-1]) if conflict else (keys[1:] ^ keys[:-1]) >> OBJ_BITS
    new = torch.ones(len(keys), dtype=torch.bool, device=DEV)
    new[1:] = (same != 0) | (owner[1:] != owner[:-1])
    keys, owner = keys[new], owner[new]
    offs = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    offs[1:] = torch.cumsum(torch.bincount(owner, minlength=n), 0)
    return keys.contiguous(), offs


def _host(keys, offs):
    return keys.cpu().numpy().view(np.uint64), offs.cpu().numpy().view(np.uint64)


def _references(g, case):
    n = case["genomes"]
    clusters = max(1, n // case["per_cluster"])
    anc = _Ancestors(g, clusters, case)
    cluster = torch.arange(n, device=DEV) % clusters
    keys, owner = _members(g, anc, cluster, case["sub_hi"])
    keys, offs = _finish(keys, owner, n, False)
    return anc, keys, offs


def _sketch(keys, offs, conflict=False):
    k, o = _host(keys, offs)
    return kssdgpu.Sketch(keys=k, offs=o, names=[], conflict=conflict, obj_bits=OBJ_BITS)


def _assemblies(g, anc, case, n):
    """Assemblies and fragments of 1/80 of the median length up to three times it."""
    clusters = len(anc.count)
    lo, hi = math.log(case["bp"] / 80), math.log(case["bp"] * 3)
    if case["per_cluster"] >= case["genomes"]:  # isolates of one species: whole genomes
        lo = math.log(case["bp"] / 4)
    own = torch.exp(lo + (hi - lo) * torch.rand(n, generator=g, device=DEV, dtype=torch.float64))
    cluster = torch.randint(0, clusters, (n,), generator=g, device=DEV)
    alen = anc.count[cluster].double() / PER_BP
    keys, owner = _members(g, anc, cluster, case["sub_hi"], (own / alen).float())
    extra = ((own - alen).clamp(min=0) * PER_BP).round().long()
    more, _ = _expand(torch.zeros_like(extra), extra)
    return _finish(torch.cat([keys, _keys(g, len(more))]), torch.cat([owner, more]), n, False)


def _reads(g, anc, case, n):
    """Read sets: 1 to 5 genomes each at 5 to 50 fold coverage with 0.1 to 1 % errors, the
    errors as further objects of a context or as contexts of their own."""
    clusters = len(anc.count)
    held = torch.randint(1, 6, (n,), generator=g, device=DEV)
    sample, _ = _expand(torch.zeros_like(held), held)
    cluster = torch.randint(0, clusters, (len(sample),), generator=g, device=DEV)
    keys, part = _members(g, anc, cluster, case["sub_hi"])
    cov = 5 + 45 * torch.rand(len(sample), generator=g, device=DEV)
    err = 0.001 + 0.009 * torch.rand(len(sample), generator=g, device=DEV)
    seen = torch.rand(len(keys), generator=g, device=DEV) < (1 - torch.exp(-cov * 119 / 150))[part]
    keys, part = keys[seen], part[seen]
    rate = cov * (1 - (1 - err) ** (OBJ_BITS // 2))
    count = torch.poisson(rate[part], generator=g).long()
    at, _ = _expand(torch.zeros_like(count), count)
    base = 2 * torch.randint(0, OBJ_BITS // 2, (len(at),), generator=g, device=DEV)
    sub = torch.randint(1, 4, (len(at),), generator=g, device=DEV, dtype=torch.int64)
    noise = torch.poisson(anc.count[cluster] * cov * err * (CTX_BITS // 2), generator=g).long()
    no, _ = _expand(torch.zeros_like(noise), noise)
    all_keys = torch.cat([keys, keys[at] ^ (sub << base), _keys(g, len(no))])
    owner = sample[torch.cat([part, part[at], no])]
    return _finish(all_keys, owner, n, True)


# ------------------------------------------------------------------ counters and sequence


def _counters(g, case):
    """Sketch sizes and counters of every cell of a triangle as the self join of clustered
    genomes gives them: cells of one cluster share contexts, the others none."""
    n = case["genomes"]
    clusters = max(1, n // case["per_cluster"])
    size = (_lengths(g, clusters, case["bp"], 0.37) * PER_BP).round().long()[torch.arange(n, device=DEV) % clusters]
    p = (0.001 + (case["sub_hi"] - 0.001) * torch.rand(n, generator=g, device=DEV)).double()
    q, r = torch.tril_indices(n, n, -1, device=DEV)
    pick = (q % clusters) == (r % clusters)
    q, r = q[pick], r[pick]
    keep = ((1 - p[q]) * (1 - p[r])) ** (CTX_BITS // 2)
    xny = torch.minimum(torch.poisson(size[q] * keep, generator=g).long(), size[q])
    d = p[q] + p[r]
    differ = 1 - (1 - d) ** (OBJ_BITS // 2)
    diff = torch.minimum(torch.poisson(xny * differ, generator=g).long(), xny)
    mut2 = torch.minimum(torch.poisson(diff * (1 - (1 - d) ** (OBJ_BITS // 2 - 1)), generator=g).long(), diff)
    section = diff + mut2 + torch.poisson(mut2 * d * 4, generator=g).long()
    ctx = torch.zeros(n * (n - 1) // 2, dtype=torch.int64, device=DEV)
    obj = torch.zeros_like(ctx)
    cell = q * (q - 1) // 2 + r
    ctx[cell] = xny | (mut2 << 32)
    obj[cell] = diff | (section << 32)
    return size.to(torch.int32), ctx, obj


def _sequence(case, seed):
    """FASTA record bytes: bases in both cases, runs of N, contigs of uneven lengths."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    rng = np.random.default_rng(seed)
    letters = torch.tensor(list(b"ACGT"), dtype=torch.uint8, device=DEV)
    samples = []
    for _ in range(case["samples"]):
        bp = int(case["bp"])
        seq = letters[torch.randint(0, 4, (bp,), generator=g, device=DEV)]
        at = int(rng.integers(0, bp))
        seq[at:at + bp // 50] |= 32  # a soft-masked stretch
        at = int(rng.integers(0, bp))
        seq[at:at + 100] = ord("N")
        seq = seq.cpu().numpy().tobytes()
        cuts = np.sort(rng.integers(0, bp + 1, max(0, case["contigs"] - 1)))
        cuts = [0, *cuts.tolist(), bp]
        samples.append([seq[a:b] for a, b in zip(cuts, cuts[1:])])
    return samples


# ------------------------------------------------------------------ the cases


def _buffer(rows, dtype=np.uint32, cols=10):
    return np.zeros((int(rows), cols) if cols else int(rows), dtype=dtype)


def _into(buf, got):
    """Results whose number depends on the data, in the caller's buffer, zeros behind them."""
    buf[:len(got)] = got
    buf[len(got):] = 0
    return buf


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sketch":
        return dict(case=case, samples=_sequence(case, seed),
                    keys=_buffer(case["samples"] * case["bp"] * PER_BP * 1.25 + 4096, np.uint64, 0))
    g = torch.Generator(device=DEV).manual_seed(seed)
    s = dict(case=case)
    if kind == "values":
        n = case["genomes"]
        s["size"], s["ctx"], s["obj"] = _counters(g, case)
        s["opt"] = kssdgpu.metric_opt(s=-1, zero_const=1, zero_value=0.0)
        s["value"] = torch.zeros(n * (n - 1) // 2, dtype=torch.float64, device=DEV)
        s["recheck"] = torch.zeros(3 * 65536, dtype=torch.int64, device=DEV)
        s["listed"] = torch.zeros(1, dtype=torch.int64, device=DEV)
        return s
    anc, keys, offs = _references(g, case)
    sk = _sketch(keys, offs)
    if kind == "matrix":
        s["sketch"] = sk
        return s
    n = case["genomes"]
    s["index"] = kssdgpu.Index.from_sketch(sk)
    if kind == "self":
        s["ctx"] = torch.zeros(n * (n - 1) // 2, dtype=torch.int64, device=DEV)
        s["obj"] = torch.zeros_like(s["ctx"])
        return s
    nq = case["queries"]
    if kind == "serve":  # four assemblies to a read set
        if nq < 5:
            k, o = _host(*_assemblies(g, anc, case, nq))
            s["requests"] = np.split(k, o[1:-1].astype(np.int64))
        else:
            k, o = _host(*_assemblies(g, anc, case, nq - nq // 5))
            s["requests"] = np.split(k, o[1:-1].astype(np.int64))
            k, o = _host(*_reads(g, anc, case, nq // 5))
            s["requests"] += np.split(k, o[1:-1].astype(np.int64))
        # a query meets its clusters' genomes, and now and then another by chance
        s["hits"] = [_buffer(5 * (n // len(anc.count) + 2) + 64) for _ in s["requests"]]
        s["server"] = kssdgpu.Server(s["index"], max_batch_queries=64, max_batch_keys=1 << 24, slots=2,
                                     device_budget=2 << 30)
        return s
    qkeys, qoffs = (_reads if case.get("reads") else _assemblies)(g, anc, case, nq)
    if kind == "detail":
        s["qkeys"], s["qoffs"] = _host(qkeys, qoffs)
        s["hits"] = _buffer(nq * (n // len(anc.count) + 2))
        s["qcount"] = np.diff(s["qoffs"]).astype(np.uint32)
        s["rcount"] = np.diff(sk.offs).astype(np.uint32)
        return s
    s["qkeys"], s["qoffs"] = qkeys, qoffs
    s["out"] = [torch.zeros((nq, n), dtype=torch.int64, device=DEV) for _ in range(4 if case["unique"] else 2)]
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "self":
        s["index"].self_lower_dev(s["ctx"], s["obj"])
        return s["ctx"], s["obj"]
    if kind == "matrix":
        index = kssdgpu.Index.from_sketch(s["sketch"])
        count, unique = index.ref_ctx_counts(False, False)
        ctx, obj = index.self_lower()
        index.close()
        return count, unique, ctx, obj
    if kind == "block":
        out = s["out"]
        s["index"].count_block_dev(s["qkeys"], s["qoffs"], case["queries"], *out,
                                   flags=kssdgpu.UNIQUE if case["unique"] else 0)
        return out
    if kind == "detail":
        hits, rows = s["index"].count_detail(s["qkeys"], s["qoffs"], s["qcount"], s["rcount"], kssdgpu.UNIQUE)
        return _into(s["hits"], hits.view(np.uint32).reshape(-1, 10)), rows
    if kind == "serve":
        tickets = [s["server"].submit(k) for k in s["requests"]]
        return [_into(buf, s["server"].result(t)[0].view(np.uint32).reshape(-1, 10))
                for t, buf in zip(tickets, s["hits"])]
    if kind == "sketch":
        keys, offs = kssdgpu.sketch(s["samples"])
        return _into(s["keys"], keys), offs
    n = case["genomes"]
    kssdgpu.lower_metric_dev(s["opt"], n, s["size"], s["size"], s["ctx"], s["obj"], s["value"], s["recheck"], 65536,
                             s["listed"])
    return s["value"], s["listed"]


def work(case):
    """Bytes of one pass: its inputs read once and its outputs written once, expected sizes.
    Contexts of one cluster's surviving keys are shared, the replaced ones are single."""
    kind = case["kind"]
    if kind == "sketch":
        bases = case["samples"] * float(case["bp"])
        return {"bytes": bases + 8 * bases * PER_BP, "flops": 0}
    n = case["genomes"]
    clusters = max(1, n // case["per_cluster"])
    cells = n * (n - 1) / 2
    if kind == "values":
        return {"bytes": 24 * cells + 8 * n, "flops": 0}
    keys = n * case["bp"] * PER_BP * math.exp((0.2 if clusters == 1 else 0.37) ** 2 / 2)
    hi = case["sub_hi"]
    keep = ((1 - 0.001) ** 23 - (1 - hi) ** 23) / (23 * (hi - 0.001)) * (1 - 0.001) ** 32
    shared = keys * keep  # postings in contexts of an ancestor
    contexts = keys * (1 - keep) + keys * clusters / n
    if kind == "self":
        return {"bytes": 4 * contexts + 8 * shared + 16 * cells, "flops": 0}
    if kind == "matrix":
        return {"bytes": 8 * keys + 16 * cells + 8 * n, "flops": 0}
    nq = case["queries"]
    if case["per_cluster"] >= n:
        lo, top = case["bp"] / 4, case["bp"] * 3
    else:
        lo, top = case["bp"] / 80, case["bp"] * 3
    qkeys = nq * PER_BP * (top - lo) / math.log(top / lo)
    if case.get("reads"):
        qkeys = nq * 3 * case["bp"] * PER_BP * (1 + 27.5 * 0.0055 * (10 + 22))
    # a query key, and once the 8 bytes of each posting of the contexts that it meets
    walked = min(shared, qkeys * (min(1.0, case["bp"] * PER_BP * nq / qkeys)) * keep * n / clusters * keep)
    cell = {"block": 32 if case.get("unique") else 16}.get(kind, 0)
    return {"bytes": 8 * qkeys + 8 * walked + cell * nq * n, "flops": 0}


def exact(case, seed):
    """The matrix values (lm3ways distance and the calibration trees) by numpy in 64 bits;
    the other kinds return counts and keys, which have no rounding."""
    if case["kind"] != "values":
        return None
    g = torch.Generator(device=DEV).manual_seed(seed)
    size, ctx, obj = (t.cpu().numpy() for t in _counters(g, case))
    opt = kssdgpu.metric_opt(s=-1)
    nodes = np.frombuffer((np.ctypeslib.ctypes.c_ubyte * (16 * opt.hgb_nodes_count)).from_address(opt.hgb_nodes),
                          dtype=[("x", "<f8"), ("feature", "i1"), ("flags", "u1"), ("left", "<u2"), ("right", "<u2"),
                                 ("pad", "<u2")])
    begin = np.frombuffer((np.ctypeslib.ctypes.c_uint * (opt.hgb_trees + 1)).from_address(opt.hgb_tree_begin),
                          dtype=np.uint32).astype(np.int64)
    xny, mut2 = ctx & 0xFFFFFFFF, ctx >> 32
    diff, section = obj & 0xFFFFFFFF, obj >> 32
    q, r = np.tril_indices(case["genomes"], -1)
    value = np.zeros(len(ctx))
    afq, afr = xny / size[q], xny / size[r]
    at = np.nonzero((xny > 0) & (np.maximum(afq, afr) >= 0.5))[0]
    xny, mut2, diff, section = (v[at].astype(np.float64) for v in (xny, mut2, diff, section))
    afq, afr = afq[at], afr[at]
    ani = 1.0 - _lm3ways(xny, section, mut2, diff)
    af = np.clip(afr, 1e-12, 1.0)
    aaf = np.clip(1.0 + np.log(af) / 11.0, 0, 1)
    raw = np.clip(ani, 0, 1)
    x = np.stack([raw, af, np.log1p(xny), diff / xny, section / xny, mut2 / xny, aaf, raw - aaf, af < 0.2,
                  (af >= 0.2) & (af < 0.5), af >= 0.5])
    pred = np.full(len(at), opt.hgb_baseline)
    rows = np.arange(len(at))
    for t in range(opt.hgb_trees):
        node = np.full(len(at), begin[t])
        for _ in range(64):
            nd = nodes[node]
            leaf = (nd["flags"] & 1) != 0
            if leaf.all():
                break
            left = x[np.where(leaf, 0, nd["feature"]), rows] <= nd["x"]
            node = np.where(leaf, node, begin[t] + np.where(left, nd["left"], nd["right"]))
        pred += nodes[node]["x"]
    pred = np.clip(pred, 0, 1)
    same = (diff == 0) & (section == 0) & (mut2 == 0) & (afq == 1.0) & (afr == 1.0)
    best = np.where(same, 1.0, pred)
    value[at] = np.where(best > 0, best, ani)
    return value, None


_DENOM = (1.0178887, 1.0135146, 1.0302181, 1.1205122, 1.0136223, 0.9803396, 1.0021964, 0.9839395, 0.9988935,
          0.9690589, 0.9888171, 0.9817371)
_DENOM95 = (1.0145656, 1.2708196, 1.2169829, 0.3904416, 0.8147527, 1.3389150, 2.0581364, -1.4624736, 1.6877678,
            2.4390067, 0.7878482, 0.6697437)
_COEF = (6.86905236142636, -5.85271800517096e-08, 7.43351941016881e-06, -1.95859228059721e-05, -8.44336369105416e-06,
         -11726.5478433625, -111109.682632437, 121000.895632267, -741.538955661909, -1894.53741972785,
         2585.81964981999, -7744.5216892858, -18190.2514369096, 23306.3090989115, 8352.82760552325, 19782.4294837312,
         -25518.2493259614)
_COEF95 = (-1.69173585242774, -3.64716315423252e-08, 2.85880264052975e-05, -5.5597924264054e-05,
           -2.96208613804271e-05, 1106.96550282022, -83.197177767225, -1671.88720051458, 152.75590068948,
           212.734805232395, 208.388739816682, -0.27860125939004, 2.27065806912198, -10.2977013026837,
           -250.681324281127, -403.751360812353, -137.96628693833)


def _lm3ways(X, S, M, D):
    """The lm3ways distance of the counters (scale 1: the default down-sampling)."""
    def core(p, c):
        d1 = 1 / (p[0] * X + p[1] * S + p[2] * M + p[3] * D + 1e-8)
        d2 = 1 / (p[4] * X + p[5] * S + p[6] * M + p[7] * D + 1e-8)
        d3 = 1 / (p[8] * X + p[9] * S + p[10] * M + p[11] * D + 1e-8)
        return (c[0] + c[1] * X + c[2] * S + c[3] * M + c[4] * D + c[5] * d1 + c[6] * d2 + c[7] * d3 + c[8] * X * d1
                + c[9] * S * d1 + c[10] * M * d1 + c[11] * X * d2 + c[12] * S * d2 + c[13] * M * d2 + c[14] * X * d3
                + c[15] * S * d3 + c[16] * M * d3)
    dist = core(_DENOM, _COEF)
    dist = np.where(dist < 0.05, core(_DENOM95, _COEF95), dist)
    return np.where(D <= 0, 0.0, np.maximum(dist, 0.0))
