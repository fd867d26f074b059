"""The activation entry against the plain torch restatement of perf/cases.py
where its branches change: air above, across and below the ice transition,
modes without aerosol or with none that takes up water, no updraft. The
erf arguments are sums of logs of order 30 with a rounding of 1e-15 each,
over at least 0.47 sqrt(2): 1e-13 on fractions of order one."""

import pytest
import torch

from mam4xx_b200 import workloads as wl
from perf import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncol", [1, 3, 129])
@pytest.mark.parametrize("edge", ["warm", "mixed", "cold", "no_coarse", "soot", "calm"])
def test_activation_matches_restatement(cuda_device, ncol, edge):
    s = cases.prepare({"kind": "activate", "ncol": ncol, "nlev": 43, "sky": "uniform"}, 7)
    x, w = s["x"], s["w"]
    lo, hi = {"warm": (274.0, 300.0), "mixed": (254.0, 273.0)}.get(edge, (200.0, 252.0))
    x[wl.IN_T] = torch.linspace(lo, hi, x.shape[1], dtype=torch.float64, device="cuda")
    if edge == "no_coarse":
        x[wl.IN_AER_I + 13:wl.IN_AER_I + 21] = 0.0
    if edge == "soot":  # primary carbon of black carbon alone, no number
        x[wl.IN_AER_I + 21] = x[wl.IN_AER_I + 23] = x[wl.IN_AER_I + 24] = 0.0
    if edge == "calm":
        w[::2] = 0.0
    want, got = cases._exact_activate(s), cases.run(s)
    torch.cuda.synchronize()
    for k, v in want.items():
        scale = w.abs() if k.startswith("flux") else torch.ones_like(w)
        assert got[k].shape == v.shape
        assert bool(((got[k] - v).abs() <= 1e-13 * scale).all()), k
