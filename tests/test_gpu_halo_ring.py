"""Halo form of the general 16-bit kernel (stride-1 filters of at least four taps, more than 16 channels, images of 23 rows and more):
filter slices by filter rows and by single taps, two and three halo tiles in flight, one and several tiles per image, dilation, asymmetric
padding, several channel slices, and more work than the ring holds."""
import numpy as np
import pytest
import torch

from helpers import normal, rel_err, uniform

pytestmark = pytest.mark.gpu

TOL = {"f16": 2.0 ** -10, "bf16": 2.0 ** -7}      # half a unit in the last place of max|ref|, twice for the sums' own error


# n, ci, co, h, w, kh, kw, pad (top, left, bottom, right), dilation
@pytest.mark.parametrize("dtype,case", [
    ("f16", (2, 32, 24, 24, 16, 3, 3, (1, 1, 1, 1), 1)),
    ("f16", (1, 20, 36, 33, 19, 2, 2, (0, 1, 1, 0), 1)),
    ("bf16", (1, 64, 40, 56, 24, 3, 3, (1, 1, 1, 1), 1)),
    ("f16", (1, 36, 20, 31, 17, 5, 5, (2, 2, 2, 2), 1)),
    ("bf16", (1, 96, 33, 28, 9, 5, 5, (2, 1, 2, 3), 1)),
    ("f16", (1, 18, 20, 30, 26, 7, 7, (3, 3, 3, 3), 1)),
    ("f16", (1, 24, 20, 40, 30, 3, 3, (4, 4, 4, 4), 4)),
    ("f16", (1, 24, 20, 26, 30, 1, 9, (0, 4, 0, 4), 1)),
    ("f16", (1, 24, 20, 30, 12, 9, 1, (4, 0, 4, 0), 1)),
])
def test_halo_form(oracle, dtype, case):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import gpu_util as gpu
    n, ci, co, h, w, kh, kw, pad, dil = case
    x = gpu.rounded(uniform(71, (4 * n, ci, h, w)), dtype)
    f = gpu.rounded(normal(72, (4, co, ci, kh, kw), std=(2.0 / (4 * ci * kh * kw)) ** 0.5), dtype)
    b = gpu.rounded(uniform(73, (4, co)), dtype)
    ref = oracle.conv2d_fwd(x, f, b, (1, 1), (dil, dil), pad)
    y = gpu.run_conv_fwd(x, f, b, (1, 1), pad, dtype, "16p", "tensor", dilation=(dil, dil))
    dy = gpu.rounded(normal(74, ref.shape), dtype)
    rdw, rdx = oracle.conv2d_bwd(x, f, dy, (1, 1), (dil, dil), pad)
    dw, dx = gpu.run_conv_bwd(x, f, dy, (1, 1), pad, dtype, "16p", "tensor", True, dilation=(dil, dil))
    for got, want, what in ((y, ref, "y"), (dx, rdx, "dx"), (dw, rdw, "dw")):
        assert np.all(np.isfinite(got)), what
        assert rel_err(got, want) <= TOL[dtype], (what, rel_err(got, want))
