"""The denoiser's loss beyond a warp is summed in FP64: terms whose sums are exact in a warp's
FP32 and in FP64, but not in FP32 across warps, give the exact mean."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("channels", [(16,), (32,)])
@pytest.mark.parametrize("side", [8, 24])
def test_loss_is_summed_in_64_bits(gpu, channels, side):
    import torch

    net = gpu.Denoiser(channels, seed=1)
    net.set_params(np.zeros(net.n_params, np.float32))  # predicts 0: the loss is the mean target
    n = side ** 3
    # by warps of 32 voxels: a sum of 2^25, then one of 1, which 2^25 + 1 loses in FP32
    t = np.where(np.arange(n) // 32 % 2 == 0, 2.0 ** 20, 2.0 ** -5).astype(np.float32)
    x = torch.zeros((1, side, side, side, 16), dtype=torch.bfloat16, device="cuda")
    loss = net.backward(x, torch.from_numpy(t.reshape(1, side, side, side)).cuda())
    assert loss == t.astype(np.float64).sum() / n
