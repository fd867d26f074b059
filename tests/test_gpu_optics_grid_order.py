"""Refractive-index grids in any order: the bracket of an index starts before
the first grid point above it, in the order given. Against the restatement
of perf/cases.py with a linear search, in the bounds of the tests of the
ascending grids (test_gpu_rad_bands.py)."""

import numpy as np
import pytest
import torch

from mam4xx_b200 import workloads as wl
from perf import cases

pytestmark = pytest.mark.gpu


def _first_above(grid, v):
    n = grid.numel()
    above = v[None, :] < grid[:, None]
    first = torch.where(above.any(0), above.long().argmax(0), n)
    i = (first - 1).clamp(min=0)
    j = (i + 1).clamp(max=n - 1)
    dx = grid[j] - grid[i]
    return i, j, torch.where(dx.abs() > 1e-20, (v - grid[i]) / dx, torch.zeros_like(v))


def _reorder(n, order):
    k = np.arange(n)
    if order == "descending":
        return k[::-1]
    if order == "swapped":  # one pair out of place
        k[n // 2 - 1], k[n // 2] = k[n // 2], k[n // 2 - 1]
    if order == "rotated":
        k = np.roll(k, 3)
    if order == "repeated":
        k[n // 2:] = k[n // 2 - 1:n - 1]
    return k


# the rotated grids extrapolate the shortwave fit beyond exp's range: the
# restatement itself is infinite there
@pytest.mark.parametrize("kind,order", [
    (k, o) for k in ("rad_sw", "rad_lw")
    for o in ("ascending", "descending", "swapped", "rotated", "repeated")
    if (k, o) != ("rad_sw", "rotated")])
def test_grids_in_any_order(cuda_device, monkeypatch, kind, order):
    name = "make_optics_%s_tables" % kind[4:]
    tables = getattr(wl, name)()
    for t in ("refrtab", "refitab"):
        tables[t] = np.ascontiguousarray(tables[t][..., _reorder(tables[t].shape[-1], order)])
    monkeypatch.setattr(wl, name, lambda: tables)
    monkeypatch.setattr(cases, "_bracket", _first_above)
    s = cases.prepare({"kind": kind, "ncol": 7, "nlev": 72, "sky": "uniform"}, 13)
    s["x"][wl.IN_QV] = 0.0
    got, want = cases.run(s), cases._exact_rad(s)
    torch.cuda.synchronize()
    for k, w in want.items():
        if w is not None:
            assert torch.linalg.norm(got[k] - w) <= 1e-13 * torch.linalg.norm(w), k
