"""Real-valued inputs on the general 16-bit kernel: the packed filter matrix has one component along K, and its tiled packing (whole
tiles of 32 output channels, at most nine taps) must write that one only."""
import numpy as np
import pytest
import torch

from helpers import normal, rel_err, uniform

pytestmark = pytest.mark.gpu

TOL = {"f16": 2.0 ** -10, "bf16": 2.0 ** -7}      # half a unit in the last place of max|ref|, twice for the sums' own error


@pytest.mark.parametrize("ci,co,k,stride,dtype", [(3, 64, 3, 1, "f16"), (3, 96, 3, 2, "bf16"), (65, 32, 3, 2, "f16"), (91, 128, 1, 1, "f16"),
                                                  (17, 32, 2, 1, "bf16"), (40, 64, 3, 1, "f16"), (20, 40, 3, 1, "f16"), (24, 32, 5, 1, "f16")])
def test_forward(oracle, ci, co, k, stride, dtype):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import gpu_util as gpu
    n, h, w = 3, 20, 23
    pad = (k // 2,) * 4
    x = gpu.rounded(uniform(41, (n, ci, h, w)), dtype)
    f = gpu.rounded(normal(42, (4, co, ci, k, k), std=(2.0 / (ci * k * k)) ** 0.5), dtype)
    x4 = np.concatenate([x, np.zeros((3 * n, ci, h, w), np.float32)])            # the quaternions with zero imaginary parts
    ref = oracle.conv2d_fwd(x4, f, None, (stride, stride), (1, 1), pad)
    y = gpu.run_conv_fwd(x, f, None, (stride, stride), pad, dtype, "16p", "auto", True)
    assert np.all(np.isfinite(y)) and rel_err(y, ref) <= TOL[dtype], rel_err(y, ref)
