"""The matrix-value kernel's tiling against the host epilogue, at the sizes where it can go
wrong: triangles of one cell, of less than a warp, of one warp's tile, of tiles that end
inside a row, and of full tiles; cells that take the calibration trees rare (a warp takes
each) and common (a thread takes each)."""
import ctypes as C

import numpy as np
import pytest
import torch

import kssdgpu
from test_gpu_metric import AniOpt, Feat, _host, _triangle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("opt", [dict(s=-1), dict(s=2, v=1)], ids=["calibrated", "naive"])
@pytest.mark.parametrize("n,shared", [(2, 1.0), (3, 1.0), (9, 0.5), (70, 1.0), (70, 0.02), (333, 0.3), (2200, 0.002)])
def test_values_at_tile_edges(n, shared, opt):
    host = _host()
    o = AniOpt()
    host.kssd_opt_defaults(C.byref(o))
    o.fmt = 1
    for k, v in opt.items():
        setattr(o, k, v)
    zero = C.c_double()
    zero_const = bool(host.kssd_zero_overlap_metric(C.byref(o), C.byref(zero)))
    rng = np.random.default_rng(7000 + n)
    size, q, r, lc, lo = _triangle(rng, n)
    size[size == 0] = 5001  # every cell without shared contexts takes the constant
    none = rng.random(len(lc)) >= shared
    lc[none] = 0
    lo[none] = 0
    mo = kssdgpu.metric_opt(s=o.s, e=o.e, v=int(o.v), afcut=o.afcut, drfold=o.drfold, obj_bits=o.obj_bits,
                            ctx_bits=o.ctx_bits, zero_const=int(zero_const), zero_value=zero.value)
    dev = torch.device("cuda", 0)
    up = lambda a: torch.from_numpy(a.view(np.int64 if a.dtype.itemsize == 8 else np.int32)).to(dev)  # noqa: E731
    d_size, d_lc, d_lo = up(size), up(lc), up(lo)
    # one guard word behind the values: the last tile must end with the triangle
    d_val = torch.full((len(lc) + 1,), -7.0, dtype=torch.float64, device=dev)
    d_re = torch.zeros(3 * len(lc), dtype=torch.int64, device=dev)
    d_nre = torch.zeros(1, dtype=torch.int64, device=dev)
    kssdgpu.lower_metric_dev(mo, n, d_size, d_size, d_lc, d_lo, d_val, d_re, len(lc), d_nre)
    torch.cuda.synchronize()
    got = d_val.cpu().numpy()
    assert got[-1] == -7.0
    got = got[:-1]
    re = d_re.cpu().numpy().view(kssdgpu.RECHECK_DTYPE)[:int(d_nre.item())]
    want = np.full(len(lc), zero.value)
    f = Feat()
    plain = (lc == 0) & zero_const
    for i in np.nonzero(~plain)[0]:
        c, ob = int(lc[i]), int(lo[i])
        f.XnY_ctx, f.N_mut2_ctx, f.N_diff_obj, f.N_diff_obj_section = c & 0xFFFFFFFF, c >> 32, ob & 0xFFFFFFFF, ob >> 32
        f.X_ctx = 0
        want[i] = host.kssd_pair_metric(C.byref(f), int(size[q[i]]), int(size[r[i]]), C.byref(o), None, None)
    listed = np.zeros(len(lc), dtype=bool)
    listed[re["cell"].astype(np.int64)] = True
    assert np.array_equal(np.isnan(got), listed) and listed.sum() <= len(lc) // 100
    if not opt.get("v"):  # built from + - * / alone: the host's double
        assert np.array_equal(got[~listed].view(np.uint64), want[~listed].view(np.uint64))
    assert [f"{x:f}" for x in got[~listed]] == [f"{x:f}" for x in want[~listed]]
