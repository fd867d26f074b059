"""The optics band kernels (packed tables, bracket search, volcanic values in
the same pass) against the plain torch restatement of perf/cases.py.

The fits are sums of a few dozen products of values of one sign pattern
each; relative rounding of 1e-15 per product and 60 products bound their
error by 1e-13 of the row's norm. The water uptake before them amplifies
rounding where its closed-form root cancels, which the test's cells avoid by
staying below the crystallisation humidity (no water) in all but the free
case, which is held to 1e-9.
"""

import pytest
import torch

from mam4xx_b200 import native
from mam4xx_b200 import workloads as wl
from perf import cases

pytestmark = pytest.mark.gpu


def _state(kind, ncol, nlev, edge, seed):
    s = cases.prepare({"kind": kind, "ncol": ncol, "nlev": nlev, "sky": "uniform"}, seed)
    x = s["x"]
    if edge != "free":
        x[wl.IN_QV] = 0.0
    if edge == "pure":  # single species: refractive indices at and beyond the grids' ends
        for k in range(25):
            if k not in wl.NUMBER_SLOTS and k % 3:
                x[wl.IN_AER_I + k] *= 1e-30
    if edge == "empty":
        for k in range(25):
            if k not in wl.NUMBER_SLOTS:
                x[wl.IN_AER_I + k, ::2] = 1e-60
    return s


# "empty" holds for the longwave only: the shortwave bounds the divisor of the
# refractive index by 1e-40 and then extrapolates the fit, which the
# restatement, dividing by the volume itself, does not describe
@pytest.mark.parametrize("kind,edge", [(k, e) for k in ("rad_sw", "rad_lw")
                                       for e in ("free", "dry", "pure", "empty")
                                       if (k, e) != ("rad_sw", "empty")])
@pytest.mark.parametrize("ncol,nlev", [(1, 2), (3, 33), (37, 72), (5, 129)])
def test_radiation_entries_match_restatement(cuda_device, kind, edge, ncol, nlev):
    s = _state(kind, ncol, nlev, edge, 5 + ncol)
    got, want = cases.run(s), cases._exact_rad(s)
    torch.cuda.synchronize()
    assert torch.equal(got["trop"].long(), cases._tropopause(s))
    for k, w in want.items():
        if w is None:
            continue
        scale = torch.linalg.norm(w)
        assert torch.linalg.norm(got[k] - w) <= (1e-9 if edge == "free" else 1e-13) * scale, k


@pytest.mark.parametrize("kind", ["rad_sw", "rad_lw"])
def test_plain_optics_equal_the_levels_below_the_tropopause(cuda_device, kind):
    """The entries without the volcanic aerosol run every cell; below the
    tropopause the radiation-facing ones give the same values, and the
    column optical depth does not depend on it."""
    s = _state(kind, 21, 72, "free", 9)
    ctx, n, dt = s["ctx"], s["n"], cases.DT
    got = cases.run(s)
    out = torch.zeros_like(s["out"])
    if kind == "rad_sw":
        aod = torch.zeros_like(s["aod"])
        ctx.optics_sw(s["x"].data_ptr(), n, s["pdel"].data_ptr(), out.data_ptr(), aod.data_ptr(),
                      21, 72, dt)
    else:
        ctx.optics_lw(s["x"].data_ptr(), n, s["pdel"].data_ptr(), out.data_ptr(), 21, 72, dt)
    torch.cuda.synchronize()
    below = (torch.arange(72, device="cuda")[None, :] > got["trop"][:, None]).reshape(-1)
    assert bool(below.any())
    assert torch.equal(out[:, below], s["out"][:, below])
    if kind == "rad_sw":
        assert torch.equal(aod, got["aod"])


def test_radiation_entry_without_column_depth(cuda_device):
    """aodvis may be absent: the modal stages then run the listed cells only."""
    s = _state("rad_sw", 9, 72, "free", 11)
    full = cases.run(s)
    keep = s["out"].clone()
    ctx, p = s["ctx"], lambda k: s[k].data_ptr()
    s["out"].zero_()
    ctx.aero_rad_props_sw(p("x"), s["n"], p("pdel"), p("pint"), p("zi"), p("ext"), p("ssa"),
                          p("af"), p("out"), 0, 0, 9, 72, cases.DT)
    torch.cuda.synchronize()
    assert torch.equal(keep, s["out"]) and full["trop"].numel() == 9
    assert not (ctx.last_status() & native.FLAG_NONFINITE_OUTPUT)
