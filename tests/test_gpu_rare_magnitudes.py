"""The step on states full of numbers far from their ordinary size.

The kernels take most quotients without the division's range handling and
return to the division where an operand leaves them no room (quot_in_range,
with_quotients). Here half of the gases and populations lie near the limits
of that (2^-150, 2^-450, 2^-600) or far below them, in another half of the
lanes of a warp for every field. Outputs and process tendencies equal the
restatement compiled for the GPU, which divides everywhere, bit for bit."""

import numpy as np
import pytest
import torch

from mam4xx_b200 import native
from mam4xx_b200 import workloads as wl
from oracle import pyoracle
from perf import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("low,high", [(150, 323), (30, 60), (120, 190)])
@pytest.mark.parametrize("sky", ["uneven", "uniform"])
def test_rare_magnitudes_equal_the_restatement(cuda_device, sky, low, high):
    ncol, nlev = 4000, 72
    s = cases.prepare({"kind": "slab", "ncol": ncol, "nlev": nlev, "sky": sky}, 21)
    x, n = s["x"], s["n"]
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    for row in range(wl.IN_H2SO4, native.NIN):
        r = torch.rand((2, n), generator=g, dtype=torch.float64, device="cuda")
        x[row] = torch.where(r[0] < 0.5, 10.0 ** -(low + (high - low) * r[1]), x[row])
    out = torch.full((native.NOUT, n), float("nan"), dtype=torch.float64, device="cuda")
    dg = torch.full((native.NDIAG, n), float("nan"), dtype=torch.float64, device="cuda")
    with_diag, plain = native.Context(), native.Context()
    with_diag.step([x[f].data_ptr() for f in range(native.NIN)], s["pblh"].data_ptr(),
                   [out[f].data_ptr() for f in range(native.NOUT)], ncol, nlev, cases.DT,
                   diag_ptrs=[dg[f].data_ptr() for f in range(native.NDIAG)])
    plain.step_slab(x.data_ptr(), s["pblh"].data_ptr(), s["out"].data_ptr(), n, ncol, nlev,
                    cases.DT)
    torch.cuda.synchronize()
    want, want_diag = pyoracle.GpuOracle().step(
        x.cpu().numpy(), np.full(n, 1000.0), cases.DT, diag=True)
    assert np.array_equal(dg.cpu().numpy(), want_diag, equal_nan=True)
    assert np.array_equal(out.cpu().numpy(), want, equal_nan=True)
    assert np.array_equal(s["out"].cpu().numpy(), want, equal_nan=True)
    with_diag.close()
    plain.close()
