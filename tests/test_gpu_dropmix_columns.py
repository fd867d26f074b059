"""The column kernel of dropmixnuc at the level counts where its lanes'
shares change (32 levels per lane and more), against a level-by-level NumPy
restatement. Activation comes from the library's own activation entry, on
columns of uniform temperature and pressure (so that the aerosol of the level
below is activated at the same air density).

The sub-steps are a contraction: each adds a rounding of some 10 eps of the
amounts, so nsub <= 1000 sub-steps stay within 1000 * 10 * 2e-16 = 2e-12 of
the population's largest amount."""

import numpy as np
import pytest
import torch

from mam4xx_b200 import native
from mam4xx_b200.workloads import IN_AER_C, IN_AER_I, NUMBER_SLOTS, POPULATIONS

pytestmark = pytest.mark.gpu

T, P, RAIR, G, DT = 270.0, 8.0e4, 6.022214076e23 * 1.380649e-23 / 0.028966, 9.80616, 1800.0
MODE = [m for m, _ in POPULATIONS]


def _activate(ctx, x, rho, w):
    n = x.shape[1]
    d = [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (x, rho, w)]
    out = torch.zeros((17, n), dtype=torch.float64, device="cuda")
    ctx.activate(d[0].data_ptr(), n, d[1].data_ptr(), d[2].data_ptr(), out.data_ptr(), 1, n)
    torch.cuda.synchronize()
    return out.cpu().numpy()


def _column(ctx, x, mix, pint, kvh, top, vmix):
    """One column (dropmixnuc of src/mam4xx/ndrop.hpp:1393-1714)."""
    n = x.shape[1]
    cs = x[1] / (RAIR * x[0])
    pdel, cldo, nc, wsub = mix
    cldn, wtke = x[4], np.maximum(wsub, 0.1)
    own = _activate(ctx, x, cs, wtke)
    low = x.copy()
    low[:, :-1] = x[:, 1:]
    base = _activate(ctx, low, cs, wtke)
    r, w = x[IN_AER_I:IN_AER_I + 25].copy(), x[IN_AER_C:IN_AER_C + 25].copy()
    dz, zn = 1.0 / (cs * G / pdel), G / pdel
    zs, eddy, csbot, ratio = (np.zeros(n) for _ in range(4))
    qc, fnum = nc.copy(), np.zeros((4, n))
    nact, mact = np.zeros((4, n)), np.zeros((4, n))
    for k in range(top, n):
        if k < n - 1:
            zs[k] = 1.0 / (x[2, k] - x[2, k + 1])
            eddy[k] = min(max(kvh[k + 1], 0.01), 100.0)
            csbot[k] = 2.0 * pint[k + 1] / (RAIR * (x[0, k] + x[0, k + 1]))
            ratio[k] = csbot[k] / cs[k]
        else:
            zs[k], csbot[k], ratio[k] = 1.0 / (x[2, k - 1] - x[2, k]), cs[k], 1.0
        d = cldn[k] - cldo[k]
        if d < 0:
            qc[k] *= 1 + d / cldo[k]
            move = w[:, k] * (d / cldo[k])
            w[:, k] += move
            r[:, k] -= move
        if d > 0.01:
            fnum[:, k] = own[0:4, k]
            for p in range(25):
                f = own[MODE[p], k] if p in NUMBER_SLOTS else own[4 + MODE[p], k]
                move = d * f * x[IN_AER_I + p, k]
                w[p, k] += move
                r[p, k] -= move
                if p in NUMBER_SLOTS:
                    qc[k] += move
    for k in range(top, n - 1):
        if cldn[k] > 0.01 and cldn[k] - cldn[k + 1] > 0.01:
            eddy[k] = wtke[k] / zs[k]
            if base[16, k] > 0:
                fnum[:, k] = base[0:4, k]
            nact[:, k] += base[8:12, k] * ratio[k] / dz[k] * (cldn[k] - cldn[k + 1])
            mact[:, k] += base[12:16, k] * ratio[k] / dz[k] * (cldn[k] - cldn[k + 1])
    for k in range(top, n - 1):
        if not cldn[k] > 0.01:
            qc[k] = 0.0
            r[:, k] += w[:, k]
            w[:, k] = 0.0
    lev = np.arange(top, n)
    kp, km = np.minimum(lev + 1, n - 1), np.maximum(lev - 1, top)
    ovp = np.where(cldn[kp] > 1e-10, np.minimum(cldn[lev] / np.maximum(cldn[kp], 1e-30), 1), 1)
    ovm = np.where(cldn[km] > 1e-10, np.minimum(cldn[lev] / np.maximum(cldn[km], 1e-30), 1), 1)
    ekp = zn[lev] * eddy[lev] * csbot[lev] * zs[lev]
    ekm = zn[lev] * eddy[lev - 1] * csbot[lev - 1] * zs[km]
    na, ma = np.minimum(nact[:, lev], ekp), np.minimum(mact[:, lev], ekp)
    dtmix = 0.9 * np.min(1.0 / (ekp + ekm)[ekp + ekm > 1e-6], initial=np.finfo(float).max)
    nsub = int(DT / dtmix + 1)
    dtmix = DT / nsub
    assert nsub <= 1000
    up, dn = kp - top, km - top
    R, W, Q = r[:, lev], w[:, lev], qc[lev]
    spare = np.zeros_like(R)  # the interstitial buffer that stays zero without mixing
    for _ in range(nsub):
        src = np.empty_like(R)
        for p in range(25):
            m = MODE[p]
            src[p] = (na if p in NUMBER_SLOTS else ma)[m] * R[p, up]
            src[p, -1] = max(0.0, R[p, -1] * na[m, -1] + W[p, -1] * na[m, -1])
        sn = sum(na[MODE[p]] * R[p, up] for p in NUMBER_SLOTS)
        sn[-1] += sum(src[p, -1] for p in NUMBER_SLOTS)
        Wn = np.maximum(W + dtmix * (src + ekp * (ovp * W[:, up] - W) + ekm * (ovm * W[:, dn] - W)), 0)
        if vmix:
            Q = np.maximum(Q + dtmix * (sn + ekp * (ovp * Q[up] - Q) + ekm * (ovm * Q[dn] - Q)), 0)
            R = np.maximum(R + dtmix * (-src + ekp * (R[:, up] - R + W[:, up] * (1 - ovp))
                                        + ekm * (R[:, dn] - R + W[:, dn] * (1 - ovm))), 0)
        else:
            R, spare = spare, R
        W = Wn
    clear = cldn[lev] == 0
    R, W, Q = np.where(clear, R + W, R), np.where(clear, 0.0, W), np.where(clear, 0.0, Q)
    full = lambda v: np.concatenate((np.zeros(v.shape[:-1] + (top,)), v), -1)  # noqa: E731
    return full((R - x[IN_AER_I:IN_AER_I + 25][:, lev]) / DT), full(W), full(Q), full(fnum[:, lev])


@pytest.mark.parametrize("vmix", [True, False])
@pytest.mark.parametrize("nlev,top", [(3, 1), (33, 1), (34, 1), (70, 6), (71, 6), (97, 1), (98, 1),
                                      (129, 1), (130, 1), (162, 1), (201, 1)])
def test_columns_match_restatement(cuda_device, nlev, top, vmix):
    rng = np.random.default_rng(nlev + top)
    ncol, n = 2, 2 * nlev
    x = np.zeros((native.NIN, n))
    x[0], x[1] = T, P
    x[2] = np.tile(np.arange(nlev)[::-1] * 400.0 + 200.0, ncol)
    x[4] = np.where(rng.uniform(size=n) < 0.3, 0.0, rng.uniform(0, 1, n))
    for p in range(25):
        v = 10.0 ** rng.uniform(*((6, 9) if p in NUMBER_SLOTS else (-12, -9)), (2, n))
        x[IN_AER_I + p], x[IN_AER_C + p] = v
    cldo = np.clip(x[4] + rng.uniform(-0.3, 0.3, n), 0.0, 1.0)
    mix = np.stack([np.full(n, 800.0), cldo, np.where(cldo > 0, 1e8, 0.0), rng.uniform(0.02, 2, n)])
    pint = np.full(ncol * (nlev + 1), P)
    kvh = 10.0 ** rng.uniform(-2, 1.5, ncol * (nlev + 1))
    ctx = native.Context()
    d = [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (x, mix, pint, kvh)]
    out = torch.full((66, n), float("nan"), dtype=torch.float64, device="cuda")
    ctx.dropmixnuc(d[0].data_ptr(), n, d[1].data_ptr(), d[2].data_ptr(), d[3].data_ptr(),
                   out.data_ptr(), ncol, nlev, top, DT, vertical_mix=vmix)
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    assert np.isfinite(got).all()
    for c in range(ncol):
        s = slice(c * nlev, (c + 1) * nlev)
        e = slice(c * (nlev + 1), (c + 1) * (nlev + 1))
        ptend, w, q, fnum = _column(ctx, x[:, s], mix[:, s], pint[e], kvh[e], top, vmix)
        for p in range(25):
            amount = max(x[IN_AER_I + p, s].max(), x[IN_AER_C + p, s].max())
            assert np.abs(got[16 + p, s] - ptend[p]).max() * DT <= 2e-12 * amount, ("ptend", p)
            assert np.abs(got[41 + p, s] - w[p]).max() <= 2e-12 * amount, ("qqcw", p)
        # droplets gain up to all four numbers
        amount = 1e8 + sum(x[IN_AER_I + p, s].max() for p in NUMBER_SLOTS)
        assert np.abs(got[0, s] - q)[top:].max() <= 2e-12 * amount
        assert np.allclose(got[6:10, s], fnum, rtol=1e-13, atol=0)
    ctx.close()
