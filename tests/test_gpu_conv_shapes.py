"""The denoiser's convolutions on grids that leave SMs idle: the brick shape goes by the grid."""
import numpy as np
import pytest

from test_gpu_denoiser import make_case, rel

pytestmark = pytest.mark.gpu

# on 152 SMs, the tcgen05 bricks (channels, z-slices) of the levels that are not on mma.sync:
SHAPES = [
    (1, 32, 32, 32),   # level 0: (16, 2)
    (2, 32, 32, 32),   # level 0: (16, 4)
    (1, 40, 24, 56),   # level 0: (16, 4), partial bricks along y and z
    (1, 64, 64, 64),   # level 1: (32, 2), level 2: (16, 2), level 3 on mma.sync
    (12, 32, 32, 32),  # level 1: (32, 4), level 2: (32, 2), level 3 4^3 voxels
    (3, 8, 8, 8),      # every level smaller than its bricks
]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_brick_shapes_match_mma_sync(gpu, shape):
    """The same parameters on the default path and on mma.sync throughout: the same
    predictions and gradients up to FP32 summation order and the bf16 roundings it moves
    (the tolerances of the full-size comparison of the two paths)."""
    torch = pytest.importorskip("torch")
    B, D, H, W = shape
    auto = gpu.Denoiser((16, 32, 64, 128), seed=4)
    ms = gpu.Denoiser((16, 32, 64, 128), seed=4, conv_path=2)
    x, t = make_case(13, B=B, D=D, H=H, W=W)
    xt = torch.tensor(x, dtype=torch.bfloat16, device="cuda")
    tt = torch.tensor(t, dtype=torch.float32, device="cuda")
    assert rel(auto.forward(xt).cpu().numpy(), ms.forward(xt).cpu().numpy()) < 1e-2
    la, lm = auto.backward(xt, tt), ms.backward(xt, tt)
    assert abs(la / lm - 1) < 1e-3
    assert rel(auto.grads(), ms.grads()) < 2e-2
    assert np.all(np.isfinite(auto.grads()))
