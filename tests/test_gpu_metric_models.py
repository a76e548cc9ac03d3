"""The matrix-value kernel on calibration models whose walks do not end on a leaf: a cycle, a
child past the model, more levels than a walk takes, such a level's child past the model, and splits
on features that there are not.
Every cell that takes the trees is left to the host, the others are valued as ever; few such
cells (the warp walks the trees of one together) and many (a thread walks its own)."""
import ctypes as C

import numpy as np
import pytest
import torch

import kssdgpu
from test_gpu_metric import _triangle

pytestmark = pytest.mark.gpu

NODE = np.dtype([("x", "<f8"), ("feature", "i1"), ("flags", "u1"), ("left", "<u2"), ("right", "<u2"), ("pad", "<u2")])


_kept = []  # every model's tables: the library knows a model by where its tables are


def _split(to):
    return (2.0, 1, 0, to, to, 0)  # the reference's AF is at most 1: always left


def _leaf(x):
    return (x, -1, 1, 0, 0, 0)


def _chain(n, end):
    return [_split(i + 1) for i in range(n)] + end


MODELS = {
    "sound": _chain(64, [_leaf(0.125)]),  # the deepest walk there is
    "cycle": [_split(1), _split(0)],
    "past": [_split(60000)],
    "deep": _chain(70, [_leaf(0.125)]),
    "deep_past": _chain(64, [_split(60000)]),
    "feature": [_split(1), (2.0, 11, 0, 2, 2, 0), _leaf(0.125)],
    "no_feature": [(2.0, -100, 0, 1, 1, 0), _leaf(0.125)],
}


def _values(n, size, lc, lo, tree, shared=True):
    """Values and listed cells of a model of three trees, the second one `tree`; without
    `shared` one too large for shared memory."""
    trees = [[_leaf(0.25)], tree, [_leaf(0.5)]]
    if not shared:
        trees.append([_leaf(0.0)] * 20000)
    nodes = np.array(sum(trees, []), dtype=NODE)
    begin = np.cumsum([0] + [len(t) for t in trees]).astype(np.uint32)
    _kept.append((nodes, begin))
    opt = kssdgpu.metric_opt(s=-1, zero_const=1, zero_value=0.0)
    opt.hgb_nodes, opt.hgb_nodes_count = nodes.ctypes.data, len(nodes)
    opt.hgb_tree_begin, opt.hgb_trees, opt.hgb_baseline = begin.ctypes.data, len(trees), 0.0625
    dev = torch.device("cuda", 0)
    up = lambda a: torch.from_numpy(a.view(np.int64 if a.dtype.itemsize == 8 else np.int32)).to(dev)  # noqa: E731
    d_size, d_lc, d_lo = up(size), up(lc), up(lo)
    d_val = torch.full((len(lc),), -7.0, dtype=torch.float64, device=dev)
    d_re = torch.zeros(3 * len(lc), dtype=torch.int64, device=dev)
    d_nre = torch.zeros(1, dtype=torch.int64, device=dev)
    kssdgpu.lower_metric_dev(opt, n, d_size, d_size, d_lc, d_lo, d_val, d_re, len(lc), d_nre)
    torch.cuda.synchronize()
    listed = np.zeros(len(lc), dtype=bool)
    listed[d_re.cpu().numpy().view(kssdgpu.RECHECK_DTYPE)["cell"][:int(d_nre.item())].astype(np.int64)] = True
    return d_val.cpu().numpy(), listed


@pytest.mark.parametrize("shared", [True, False])
@pytest.mark.parametrize("n,few", [(9, False), (70, False), (70, True)])
@pytest.mark.parametrize("model", list(MODELS))
def test_models(model, n, few, shared):
    rng = np.random.default_rng(100 + n)
    size, q, r, lc, lo = _triangle(rng, n)
    if few:
        none = rng.random(len(lc)) >= 0.05
        lc[none] = 0
        lo[none] = 0
    xny = (lc & np.uint64(0xFFFFFFFF)).astype(np.float64)
    sq, sr = size[q].astype(np.float64), size[r].astype(np.float64)
    with np.errstate(divide="ignore", invalid="ignore"):
        aq, ar = xny / sq, xny / sr
    same = (lo == 0) & (lc >> np.uint64(32) == 0) & (aq == 1.0) & (ar == 1.0)
    tree = (sq > 0) & (sr > 0) & (xny > 0) & (np.maximum(aq, ar) >= 0.5) & ~same
    assert tree.any()
    none, unlisted = _values(n, size, lc, lo, [_leaf(0.125)], shared)
    assert not unlisted.any()
    got, listed = _values(n, size, lc, lo, MODELS[model], shared)
    if model == "sound":  # the leaves' sum
        assert not listed.any() and (got[tree] == 0.0625 + 0.25 + 0.125 + 0.5).all()
    else:
        assert np.array_equal(listed, tree) and np.isnan(got[tree]).all()
    assert np.array_equal(got[~tree].view(np.uint64), none[~tree].view(np.uint64))
