"""MIXED_FAST runs its SOA loops with 64 registers where the batch is large
enough for a thread per loop: the values do not depend on that."""

import numpy as np
import pytest
import torch

from mam4xx_b200 import native
from mam4xx_b200.workloads import make_workload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncol", [3, 7400])  # four lanes to a long loop; a thread per loop
def test_fast_solver_shape_does_not_change_results(cuda_device, ncol):
    w = make_workload("c2", ncol=ncol, seed=3)
    x = torch.from_numpy(np.ascontiguousarray(w["in_slab"])).cuda()
    pb = torch.from_numpy(np.ascontiguousarray(w["pblh"])).cuda()
    got = []
    for regs, block in ((128, 128), (64, 256)):
        ctx = native.Context()
        t = native.default_tuning()
        t.soa_regs, t.soa_block = regs, block
        ctx.set_tuning(t)
        out = torch.full((native.NOUT, x.shape[1]), float("nan"), dtype=torch.float64,
                         device="cuda")
        ctx.step_slab(x.data_ptr(), pb.data_ptr(), out.data_ptr(), x.shape[1], w["ncol"],
                      w["nlev"], w["dt"], precision=native.MIXED_FAST)
        torch.cuda.synchronize()
        got.append(out)
        ctx.close()
    assert torch.equal(*got) and bool(torch.isfinite(got[0]).all())
