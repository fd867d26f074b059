"""Which solver kernel MIXED_FAST runs in a large batch: the caller's launch
shape as it is set, the 64-register one where the caller has set none."""

import pytest
import torch

from mam4xx_b200 import native
from perf import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("regs", [None, 64, 96, 128])
def test_solver_registers_are_the_callers(cuda_device, regs):
    from torch.profiler import ProfilerActivity, profile
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    ncol = 3500 * sms // 72 + 1  # a thread per loop
    s = cases.prepare({"kind": "mixed", "ncol": ncol, "nlev": 72, "sky": "uneven"}, 2)
    ctx = native.Context()
    if regs:
        t = native.default_tuning()
        t.soa_regs = regs
        ctx.set_tuning(t)
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        ctx.step_slab(s["x"].data_ptr(), s["pblh"].data_ptr(), s["out"].data_ptr(), s["n"], ncol,
                      72, cases.DT, precision=native.MIXED_FAST)
        torch.cuda.synchronize()
    ctx.close()
    names = [e.name.replace(" ", "") for e in prof.events() if "soa_kernel" in e.name]
    if not names:
        pytest.skip("no kernel names from the profiler")
    assert len(names) == 1 and "soa_kernel<2,%d>" % (regs or 64) in names[0]
