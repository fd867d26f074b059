"""The stages of the step with chemistry.

1. What condensation does not reach -- sizes, cloud-borne tendencies, the
   chemistry gases, and every tendency of a cell cloudy throughout -- equals
   bit for bit what the step without condensation gives, which runs a cell
   start to end in one thread: at the edges of blocks, for every cloudiness,
   and with a negative gas, which the first gas-phase step does not solve.
2. Gas-phase chemistry against a plain Python restatement of imp_sol, cells
   that converge at once and cells that need its step control alike. Both
   round alike but for the last bits of exp, pow and log10: 1e-12."""

import math

import numpy as np
import pytest
import torch

from mam4xx_b200 import native
from mam4xx_b200.workloads import (IN_CLD, IN_H2SO4, make_chem_step_inputs,
                                   make_gas_chemistry_inputs)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("optaa", [1, 2])
@pytest.mark.parametrize("ncol,nlev", [(1, 1), (7, 9), (13, 5), (3, 85), (16, 72), (37, 31)])
def test_stages_equal_one_kernel(cuda_device, ncol, nlev, optaa):
    w = make_chem_step_inputs("c2", ncol=ncol, nlev=nlev)
    x = np.ascontiguousarray(w["in_slab"])
    n = x.shape[1]
    kind = np.arange(n) % 5  # clear, nearly clear, partly, nearly cloudy, cloudy
    x[IN_CLD] = np.choose(kind, [0.0, 0.99e-5, 0.4, 0.999, 1.0])
    x[IN_H2SO4, ::7] *= -1.0
    x, pb, ch = (torch.from_numpy(np.ascontiguousarray(v)).cuda()
                 for v in (x, w["pblh"], w["chem_in"]))
    got = []
    for cond in (1, 0):
        ctx = native.Context(native.default_config(do_cond=cond, gaexch_h2so4_uptake_optaa=optaa))
        out = torch.full((native.NOUT, n), float("nan"), dtype=torch.float64, device="cuda")
        cout = torch.full((native.CHEM_NOUT, n), float("nan"), dtype=torch.float64, device="cuda")
        ctx.step_chem_slab(x.data_ptr(), pb.data_ptr(), ch.data_ptr(), out.data_ptr(),
                           cout.data_ptr(), n, ncol, nlev, w["dt"])
        torch.cuda.synchronize()
        assert ctx.last_status() & 0x5 == 0
        got.append((out.cpu().numpy(), cout.cpu().numpy()))
        ctx.close()
    (out, cout), (ref, rout) = got
    np.testing.assert_array_equal(cout, rout)
    np.testing.assert_array_equal(out[27:52], ref[27:52])
    np.testing.assert_array_equal(out[52:], ref[52:])
    cloudy = kind == 4
    np.testing.assert_array_equal(out[:, cloudy], ref[:, cloudy])


def _rates(t, photo, inv):
    m = inv[0]
    fc = 3.0e-31 * (300.0 / t) ** 3.3
    lg = math.log10(fc * m / 1.5e-12)
    so2 = fc * m / (1.0 + fc * m / 1.5e-12) * 0.6 ** (1.0 / (1.0 + lg * lg))
    dms = 1.7e-42 * math.exp(7810.0 / t) * m * 0.21 / (
        1.0 + 5.5e-31 * math.exp(7460.0 / t) * m * 0.21)
    ho2 = ((3.5e-13 * math.exp(430.0 / t) + 1.7e-33 * m * math.exp(1000.0 / t))
           * (1.0 + 1.4e-21 * inv[3] * math.exp(2200.0 / t)))
    return [photo, ho2 * (inv[6] * inv[6] / m), 2.9e-12 * math.exp(-160.0 / t) * inv[4],
            so2 * inv[4], 9.6e-12 * math.exp(-234.0 / t) * inv[4], dms * inv[4],
            1.9e-13 * math.exp(520.0 / t) * inv[5]]


_EXT = {2: 0, 4: 8, 5: 1, 12: 5, 13: 2, 17: 6, 26: 3, 27: 4, 29: 7}


def _imp_sol(delt, t, photo, ext, inv, het, y):
    """Implicit species k is tracer k + 1; SO2 -> H2SO4 and DMS -> SO2 couple."""
    r = _rates(t, photo, inv)
    loss = [het[k + 1] for k in range(30)]
    loss[0] += r[0] + r[2]
    loss[2] += r[3]
    loss[3] += r[4] + r[5] + r[6]
    c12, c23 = r[3], r[4] + 0.5 * r[5] + r[6]
    prod = [r[1]] + [ext[_EXT[k]] / inv[0] if k in _EXT else 0.0 for k in range(1, 30)]
    y, dt, done, cuts, good, steps = list(y), delt, 0.0, 0, 0, 0
    while steps < 1000:
        steps += 1
        term = [y[k + 1] / dt + prod[k] for k in range(30)]
        ok = False
        for it in range(11):
            f = [y[k + 1] / dt - (term[k] - loss[k] * y[k + 1]) for k in range(30)]
            f[1] -= c12 * y[3]
            f[2] -= c23 * y[4]
            f[3] /= -loss[3] - 1.0 / dt
            f[2] = (f[2] - c23 * f[3]) / (-loss[2] - 1.0 / dt)
            f[1] = (f[1] - c12 * f[2]) / (-loss[1] - 1.0 / dt)
            for k in [0] + list(range(4, 30)):
                f[k] /= -loss[k] - 1.0 / dt
            for k in range(30):
                y[k + 1] = max(y[k + 1] + f[k], 0.0)
            if it and all(abs(f[k]) <= 1e-40 or abs(f[k]) <= 1e-3 * y[k + 1] for k in range(30)):
                ok = True
                break
        if not ok:
            good = 0
            if cuts < 5:
                cuts += 1
                dt *= 0.5 if cuts < 5 else 0.1
        done += dt
        if abs(delt - done) <= 1e-4:
            break
        good += ok
        if good >= 2:
            dt, good = dt * 2.0, 0
        dt = min(dt, delt - done)
    return y, steps


@pytest.mark.parametrize("ncol,neg", [(1, 0.0), (2, 0.2)])
def test_gas_chemistry_matches_restatement(cuda_device, ncol, neg):
    d = make_gas_chemistry_inputs("c2", ncol=ncol, seed=3, negative_frac=neg)
    n = d["qq"].shape[1]
    keys = ("temp", "photo", "extfrc", "inv", "het", "qq")
    dev = {k: torch.from_numpy(np.ascontiguousarray(d[k])).cuda() for k in keys}
    ctx = native.Context()
    ctx.gas_chemistry(*[dev[k].data_ptr() for k in keys], n, d["ncol"], d["nlev"], d["dt"])
    torch.cuda.synchronize()
    got = dev["qq"].cpu().numpy()
    steps = set()
    for c in range(n):
        want, s = _imp_sol(d["dt"], d["temp"][c], d["photo"][c], d["extfrc"][:, c],
                           d["inv"][:, c], d["het"][:, c], d["qq"][:, c])
        steps.add(s > 1)
        np.testing.assert_allclose(got[1:, c], want[1:], rtol=1e-12, atol=1e-40)
    assert steps == ({False, True} if neg else {False})
    ctx.close()
