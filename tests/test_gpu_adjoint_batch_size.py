"""The gradient of a cell does not depend on the batch it is in: small batches
reverse their long SOA loops four lanes to a loop, large ones a loop per
thread, with every sum in the same order. The smallest batch, one that ends
inside a warp's eight loops and one of several blocks, against the first
columns of a batch on the other side of the rule, bit for bit."""

import pytest
import torch

from mam4xx_b200 import native
from perf import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [native.FP64, native.MIXED])
def test_gradient_does_not_depend_on_the_batch(cuda_device, precision):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    nlev = 72
    ncol = 3500 * sms // nlev + 1  # a loop per thread
    s = cases.prepare({"kind": "adjoint", "ncol": ncol, "nlev": nlev, "sky": "uniform"}, 31)

    def gradient(cols):
        n = cols * nlev
        x, ybar = s["x"][:, :n].contiguous(), s["ybar"][:, :n].contiguous()
        xbar = torch.full_like(x, float("nan"))
        s["ctx"].adjoint_slab(x.data_ptr(), s["pblh"].data_ptr(), ybar.data_ptr(),
                              xbar.data_ptr(), n, cols, nlev, cases.DT, precision=precision)
        torch.cuda.synchronize()
        return xbar

    large = gradient(ncol)
    assert bool(torch.isfinite(large).all())
    for cols in (1, 37, 1024):
        assert torch.equal(gradient(cols), large[:, :cols * nlev]), cols
