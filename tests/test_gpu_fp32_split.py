"""fp32 convolutions on the tensor cores: hi * hi in TF32 and the two cross terms in bf16, with accumulators of their own. The forms of the
kernels (halo tiles; 128 and 256 columns; one and several chunks of the K loop; filter gradients on pairs of SMs and on single ones), the
exponent range (the split may neither overflow nor lose small tensors), and the 16-bit filter gradient on pairs of SMs."""
import numpy as np
import pytest
import torch

from helpers import normal, rel_err, uniform

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import gpu_util
    return gpu_util


def _check(gpu, oracle, dtype, tol, n, ci, co, h, w, kh, kw, stride=(1, 1), pad=None, dil=1):
    pad = pad or ((kh - 1) * dil // 2, (kw - 1) * dil // 2, (kh - 1) * dil // 2, (kw - 1) * dil // 2)
    x = gpu.rounded(uniform(61, (4 * n, ci, h, w)), dtype)
    f = gpu.rounded(normal(62, (4, co, ci, kh, kw), std=(2.0 / (4 * ci * kh * kw)) ** 0.5), dtype)
    b = gpu.rounded(uniform(63, (4, co)), dtype)
    ref = oracle.conv2d_fwd(x, f, b, stride, (dil, dil), pad)
    y = gpu.run_conv_fwd(x, f, b, stride, pad, dtype, "16p", "tensor", dilation=(dil, dil))
    dy = gpu.rounded(normal(64, ref.shape), dtype)
    rdw, rdx = oracle.conv2d_bwd(x, f, dy, stride, (dil, dil), pad)
    dw, dx = gpu.run_conv_bwd(x, f, dy, stride, pad, dtype, "16p", "tensor", True, dilation=(dil, dil))
    for got, want, what in ((y, ref, "y"), (dx, rdx, "dx"), (dw, rdw, "dw")):
        assert np.all(np.isfinite(got)), what
        assert rel_err(got, want) <= tol, (what, rel_err(got, want))


# n, ci, co, h, w, kh, kw: halo tiles of 24 to 32 rows with aligned and unaligned rows, one and several chunks, several row tiles; plain tiles of
# both widths; filter gradients of one to four row tiles (pairs for two and four) and of one to three column tiles
@pytest.mark.parametrize("case", [(16, 32, 32, 24, 32, 3, 3), (8, 48, 40, 31, 21, 3, 3), (6, 16, 36, 56, 26, 2, 2), (5, 24, 33, 28, 30, 5, 3), (3, 100, 64, 14, 15, 3, 3),
                                  (2, 33, 96, 9, 8, 1, 1), (40, 8, 8, 16, 16, 1, 1), (2, 72, 130, 7, 7, 3, 3), (9, 130, 72, 6, 5, 1, 1)])
def test_fp32_forms(gpu, oracle, case):
    _check(gpu, oracle, "f32", gpu.TOL["f32"], *case)


def test_fp32_dilated_and_strided(gpu, oracle):
    _check(gpu, oracle, "f32", gpu.TOL["f32"], 6, 20, 36, 36, 25, 3, 3, dil=2)
    _check(gpu, oracle, "f32", gpu.TOL["f32"], 2, 40, 68, 15, 18, 3, 3, stride=(2, 2), pad=(1, 0, 0, 1))


@pytest.mark.parametrize("dtype,tol", [("f16", 2.0 ** -10), ("bf16", 2.0 ** -7)])
@pytest.mark.parametrize("case", [(2, 64, 64, 9, 11, 3, 3), (3, 40, 72, 8, 8, 3, 3), (2, 200, 130, 5, 6, 1, 1), (1, 72, 40, 7, 7, 3, 3), (2, 130, 256, 4, 5, 1, 1)])
def test_filter_gradient_row_tiles(gpu, oracle, dtype, tol, case):
    _check(gpu, oracle, dtype, tol, *case)


# Powers of two scale every product exactly, so the results are those of the unscaled tensors, scaled, as long as the low parts (2^-12 of a
# value and less) stay normal numbers: filters of 2^-103, whose low parts are 2^-115 and some octaves less. Further down the low parts are
# lost one by one, as they were with three TF32 products (2^-116: 2e-5, before 6e-6).
@pytest.mark.parametrize("ex,ew", [(100, -100), (-100, 90), (60, 40)])
def test_fp32_exponent_range(gpu, ex, ew):
    n, ci, co, h, w = 4, 20, 24, 26, 17
    x, f, dy = uniform(65, (4 * n, ci, h, w)), normal(66, (4, co, ci, 3, 3), std=0.1), uniform(67, (4 * n, co, h, w))
    x[0, 0], f[1] = 0.0, 0.0
    pad = (1, 1, 1, 1)
    sx, sw = np.float32(2.0 ** ex), np.float32(2.0 ** ew)
    y = gpu.run_conv_fwd(x, f, None, (1, 1), pad, "f32", "16p", "tensor")
    ys = gpu.run_conv_fwd(x * sx, f * sw, None, (1, 1), pad, "f32", "16p", "tensor")
    assert rel_err(ys * np.float32(2.0 ** -(ex + ew)), y) <= 2.0 ** -22
    dw, _ = gpu.run_conv_bwd(x, f, dy, (1, 1), pad, "f32", "16p", "tensor", True)
    dws, _ = gpu.run_conv_bwd(x * sx, f, dy * sw, (1, 1), pad, "f32", "16p", "tensor", True)
    # (split reductions add in any order: a few units in the last place of the largest)
    assert rel_err(dws * np.float32(2.0 ** -(ex + ew)), dw) <= 2e-6


def test_fp32_values_next_to_the_largest(gpu):
    # a pointwise layer whose input rounds to infinity in TF32 and in bf16: 3.4e38 * 2^-20 has to come out finite
    big = np.float32(3.4028e38)
    x = np.zeros((4, 20, 8, 8), np.float32)
    x[0, 3] = big
    f = np.zeros((4, 24, 20, 1, 1), np.float32)
    f[0, 5, 3] = np.float32(2.0 ** -20 * 1.2345678)
    y = gpu.run_conv_fwd(x, f, None, (1, 1), (0, 0, 0, 0), "f32", "16p", "tensor")
    want = np.float64(big) * np.float64(f[0, 5, 3, 0, 0])
    assert np.all(np.isfinite(y))
    assert np.max(np.abs(y[0, 5] / want - 1)) <= 4e-6
    x[0, 3, 0, 0] = np.inf
    assert not np.isfinite(gpu.run_conv_fwd(x, f, None, (1, 1), (0, 0, 0, 0), "f32", "16p", "tensor")[0, 5, 0, 0])
