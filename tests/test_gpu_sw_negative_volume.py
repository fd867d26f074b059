"""Shortwave optics of modes whose dry volume is slightly below zero, as
advection leaves it: the reference returns before any arithmetic, so such a
mode adds nothing to any band. The outputs are those of the same cells with
the mode's masses at zero, whose products are zeros too, bit for bit."""

import pytest
import torch

from mam4xx_b200 import workloads as wl
from perf import cases

pytestmark = pytest.mark.gpu


def _run(s, radiation):
    if radiation:
        cases.run(s)
    else:
        s["trop"].zero_()
        s["ctx"].optics_sw(s["x"].data_ptr(), s["n"], s["pdel"].data_ptr(), s["out"].data_ptr(),
                           s["aod"].data_ptr(), s["ncol"], s["nlev"], cases.DT)
    torch.cuda.synchronize()
    return s["out"].clone(), s["aod"].clone()


@pytest.mark.parametrize("radiation", [True, False])
@pytest.mark.parametrize("humid", [True, False])
@pytest.mark.parametrize("modes", [(0,), (1,), (2,), (3,), (0, 1, 2, 3)])
@pytest.mark.parametrize("mass", [-1e-36, -1e-30, -1e-20, -1e-15])
def test_slightly_negative_mode_adds_nothing(cuda_device, radiation, humid, modes, mass):
    s = cases.prepare({"kind": "rad_sw", "ncol": 5, "nlev": 37, "sky": "uniform"}, 3)
    x = s["x"]
    if not humid:
        x[wl.IN_QV] = 0.0
    rows = [wl.IN_AER_I + k for m in modes for k in wl.MODE_SPECIES_SLOTS[m]]
    x[rows, ::2] = 0.0
    want = _run(s, radiation)
    x[rows, ::2] = mass
    got = _run(s, radiation)
    for w, g in zip(want, got):
        assert bool(torch.isfinite(w).all()) and torch.equal(w, g)


def test_single_negative_species(cuda_device):
    """One species below zero and the others absent."""
    s = cases.prepare({"kind": "rad_sw", "ncol": 3, "nlev": 72, "sky": "uniform"}, 4)
    x = s["x"]
    for m in range(4):
        x[[wl.IN_AER_I + k for k in wl.MODE_SPECIES_SLOTS[m]]] = 0.0
    want = _run(s, True)
    for m in range(4):
        slots = wl.MODE_SPECIES_SLOTS[m]
        x[wl.IN_AER_I + slots[len(slots) // 2]] = -1e-19
    got = _run(s, True)
    for w, g in zip(want, got):
        assert bool(torch.isfinite(w).all()) and torch.equal(w, g)
