"""The step with process tendencies in stages against the same step in one
thread per cell, which is what a stream under capture runs: bit for bit, for
batches at the edges of blocks, cells of every cloudiness, absent fields and
every process switch."""

import numpy as np
import pytest
import torch

from mam4xx_b200 import native
from mam4xx_b200.workloads import IN_CLD, make_workload

pytestmark = pytest.mark.gpu


def _call(ctx, x, pb, ncol, nlev, absent, stream=0):
    n = x.shape[1]
    out = torch.full((native.NOUT, n), float("nan"), dtype=torch.float64, device="cuda")
    dg = torch.full((native.NDIAG, n), float("nan"), dtype=torch.float64, device="cuda")

    def step():
        ctx.step([x[f].data_ptr() for f in range(native.NIN)], pb.data_ptr(),
                 [out[f].data_ptr() for f in range(native.NOUT)], ncol, nlev, 1800.0,
                 diag_ptrs=[None if absent and f % absent == 0 else dg[f].data_ptr()
                            for f in range(native.NDIAG)], stream=stream)
    return out, dg, step


@pytest.mark.parametrize("cfg", [{}, dict(do_rename=0), dict(do_newnuc=0), dict(do_coag=0),
                                 dict(gaexch_h2so4_uptake_optaa=1)])
@pytest.mark.parametrize("ncol,nlev,absent", [(1, 1, 0), (7, 9, 3), (13, 5, 2), (16, 72, 0),
                                              (37, 31, 7)])
def test_stages_equal_one_kernel(cuda_device, cfg, ncol, nlev, absent):
    full = native.default_config()
    for k, v in cfg.items():
        setattr(full, k, v)
    w = make_workload("c2", ncol=ncol, nlev=nlev, seed=ncol)
    x = np.ascontiguousarray(w["in_slab"])
    kind = np.arange(x.shape[1]) % 5  # clear, nearly clear, partly, nearly cloudy, cloudy
    x[IN_CLD] = np.choose(kind, [0.0, 0.99e-5, 0.4, 0.999, 1.0])
    x = torch.from_numpy(x).cuda()
    pb = torch.from_numpy(w["pblh"]).cuda()
    ctx = native.Context(full)
    out, dg, step = _call(ctx, x, pb, ncol, nlev, absent)
    before = ctx.launch_count()
    step()
    torch.cuda.synchronize()
    assert ctx.launch_count() - before == 6
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    ref, rdg, step = _call(ctx, x, pb, ncol, nlev, absent, s.cuda_stream)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        step()
    g.replay()
    torch.cuda.synchronize()
    assert ctx.launch_count() - before == 7
    assert torch.equal(out, ref) and bool(torch.isfinite(out).all())
    assert torch.equal(dg.nan_to_num(nan=-1.0), rdg.nan_to_num(nan=-1.0))
    written = torch.isfinite(dg).all(1).cpu().numpy()
    assert np.array_equal(written, [not (absent and f % absent == 0) for f in range(native.NDIAG)])
    del g
    ctx.close()
