"""The radiation-facing optics under stream capture, in a context whose only
call of the size was the plain optics entry: nothing is allocated (which a
capture forbids), and the replayed graph gives what a direct call gives."""

import pytest
import torch

from mam4xx_b200 import native
from mam4xx_b200 import workloads as wl
from perf import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["rad_sw", "rad_lw"])
def test_capture_after_the_plain_entry(cuda_device, kind):
    ncol, nlev = 13, 37
    s = cases.prepare({"kind": kind, "ncol": ncol, "nlev": nlev, "sky": "uniform"}, 17)
    cases.run(s)
    torch.cuda.synchronize()
    keys = [k for k in ("out", "aod", "trop") if k in s]
    want = {k: s[k].clone() for k in keys}
    ctx = s["ctx"] = native.Context()
    p = lambda k: s[k].data_ptr()  # noqa: E731
    if kind == "rad_sw":
        ctx.optics_sw_set_tables(wl.make_optics_sw_tables())
        ctx.optics_sw(p("x"), s["n"], p("pdel"), p("out"), p("aod"), ncol, nlev, cases.DT)
    else:
        ctx.optics_lw_set_tables(wl.make_optics_lw_tables())
        ctx.optics_lw(p("x"), s["n"], p("pdel"), p("out"), ncol, nlev, cases.DT)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        cases.run(s)
    for k in keys:
        s[k].zero_()
    graph.replay()
    torch.cuda.synchronize()
    for k in keys:
        assert torch.equal(s[k], want[k]), k
    del graph
    ctx.close()
