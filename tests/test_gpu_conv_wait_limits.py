"""The tcgen05 convolution under small wait limits: whichever of its warps' lanes see a phase
before their polls run out, every CTA ends, the call reports the device error or gives the
result of the default limit, and the network works on afterwards."""
import numpy as np
import pytest

from opendxmc_gb300 import native as N
from test_gpu_denoiser import make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("polls", [1, 2, 3, 16, 64, 65, 1024])
def test_every_cta_ends_whatever_its_lanes_saw(gpu, polls):
    import torch

    net = gpu.Denoiser((16, 32, 64), seed=2, conv_path=1)
    x, t = make_case(17, B=2, D=24, H=40, W=16)  # no brick shape fills these edges
    xt = torch.tensor(x, dtype=torch.bfloat16, device="cuda")
    tt = torch.tensor(t, dtype=torch.float32, device="cuda")
    ref = net.forward(xt).cpu().numpy()
    loss = net.backward(xt, tt)
    for _ in range(3):
        net.set_wait_limit(polls)
        try:
            assert net.backward(xt, tt) == pytest.approx(loss, rel=1e-9)
        except N.DxmcgError as err:
            assert err.code == -5
        net.set_wait_limit(0)
        np.testing.assert_array_equal(net.forward(xt).cpu().numpy(), ref)
    assert net.backward(xt, tt) == pytest.approx(loss, rel=1e-9)
