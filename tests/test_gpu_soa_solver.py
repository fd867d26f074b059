"""The SOA solver's forms give the reference arithmetic bit for bit: four
lanes per long loop (small batches), one lane per loop (large ones), the
quotients of moderate operands and the division for all others.

The restatement compiled for the GPU (oracle/libmam4oracle_gpu.so) computes
every loop with plain divisions; equality is exact, so no tolerance enters.
"""

import numpy as np
import pytest
import torch

from mam4xx_b200 import native
from mam4xx_b200.workloads import IN_AER_I, make_workload, pblh_per_cell
from oracle.pyoracle import GpuOracle

pytestmark = pytest.mark.gpu

SOA_SLOTS = (2, 9, 18)  # SOA of the accumulation, aitken and coarse modes


def _step(ctx, x, pb, ncol, nlev, dt, precision=native.FP64):
    out = torch.full((native.NOUT, x.shape[1]), float("nan"), dtype=torch.float64, device="cuda")
    ctx.step_slab(x.data_ptr(), pb.data_ptr(), out.data_ptr(), x.shape[1], ncol, nlev, dt,
                  precision=precision)
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("soa,gas", [(1.0, 1.0), (0.0, 1.0), (1e-42, 1e-40), (1e-300, 1e-290),
                                     (1e40, 1e30)])
@pytest.mark.parametrize("name", ["c1", "c2", "c4"])
def test_states_in_and_out_of_the_quotients_range(cuda_device, name, soa, gas):
    """Particle SOA and SOA gas scaled to zero, below and above the range
    in which the solver replaces the division."""
    w = make_workload(name, ncol=8 if name == "c1" else 40, seed=77)
    x = w["in_slab"]
    for s in SOA_SLOTS:
        x[IN_AER_I + s, ::2] *= soa
    x[6, ::3] *= gas
    ctx = native.Context()
    got = _step(ctx, torch.from_numpy(x).cuda(), torch.from_numpy(w["pblh"]).cuda(), w["ncol"],
                w["nlev"], w["dt"]).cpu().numpy()
    ctx.close()
    ref = GpuOracle().step(x, pblh_per_cell(w), w["dt"])
    assert np.array_equal(got, ref, equal_nan=True)


@pytest.mark.parametrize("dt", [1.0, 1800.0, 86400.0])
def test_step_lengths(cuda_device, dt):
    """Loops of one second, of the usual step, and long steps that
    meet the cap of 1,000 passes."""
    w = make_workload("c2", ncol=24, seed=78)
    ctx = native.Context()
    got = _step(ctx, torch.from_numpy(w["in_slab"]).cuda(), torch.from_numpy(w["pblh"]).cuda(),
                w["ncol"], w["nlev"], dt).cpu().numpy()
    ctx.close()
    ref = GpuOracle().step(w["in_slab"], pblh_per_cell(w), dt)
    assert np.array_equal(got, ref, equal_nan=True)


@pytest.mark.parametrize("precision", [native.FP64, native.MIXED, native.MIXED_FAST])
def test_small_and_large_batches_agree(cuda_device, precision):
    """The same cells alone (four lanes per long loop) and repeated until
    the batch takes one lane per loop."""
    w = make_workload("c2", ncol=64, seed=79)
    x, pb = torch.from_numpy(w["in_slab"]).cuda(), torch.from_numpy(w["pblh"]).cuda()
    n, sms = x.shape[1], torch.cuda.get_device_properties(0).multi_processor_count
    times = 3500 * sms // n + 1
    ctx = native.Context()
    small = _step(ctx, x, pb, w["ncol"], w["nlev"], w["dt"], precision)
    big = _step(ctx, x.repeat(1, times), pb.repeat(times), w["ncol"] * times, w["nlev"], w["dt"],
                precision)
    ctx.close()
    assert torch.equal(big, small.repeat(1, times))


def _adjoint(ctx, x, pb, ybar, ncol, nlev, dt, precision):
    xb = torch.full((native.NIN, x.shape[1]), float("nan"), dtype=torch.float64, device="cuda")
    ctx.adjoint_slab(x.data_ptr(), pb.data_ptr(), ybar.data_ptr(), xb.data_ptr(), x.shape[1],
                     ncol, nlev, dt, precision=precision)
    torch.cuda.synchronize()
    return xb


@pytest.mark.parametrize("precision", [native.FP64, native.MIXED])
@pytest.mark.parametrize("interval", [1, 4])
def test_adjoint_of_small_and_large_batches_agrees(cuda_device, precision, interval):
    """Loops reversed on four lanes and on one. Every sum that feeds the
    reverse sweep is taken in the same order, so all gradients are equal but
    the temperature's, whose equilibrium-gas part is added up mode by mode
    and then over the modes: a reordered sum of at most 8,000 terms, within
    8,000 eps of the terms' size (2e-12), here against the row's norm."""
    w = make_workload("c2", ncol=24, seed=81)
    x, pb = torch.from_numpy(w["in_slab"]).cuda(), torch.from_numpy(w["pblh"]).cuda()
    n, sms = x.shape[1], torch.cuda.get_device_properties(0).multi_processor_count
    ybar = torch.from_numpy(np.random.default_rng(82).standard_normal((native.NOUT, n))).cuda()
    times = 3500 * sms // n + 1
    ctx = native.Context()
    ctx.set_adjoint_checkpoint(interval)
    small = _adjoint(ctx, x, pb, ybar, w["ncol"], w["nlev"], w["dt"], precision)
    big = _adjoint(ctx, x.repeat(1, times), pb.repeat(times), ybar.repeat(1, times),
                   w["ncol"] * times, w["nlev"], w["dt"], precision)[:, -n:]
    ctx.close()
    assert torch.equal(small[1:], big[1:])
    d = float(torch.linalg.norm(small[0] - big[0]) / torch.linalg.norm(big[0]))
    assert d <= 2e-12
