"""fp32 convolutions on the tensor cores: hi * hi and the two cross terms in TF32. The forms of the kernels (halo tiles; 128 and 256 columns; one and
several chunks of the K loop; filter gradients of one and several row tiles), the exponent range (the split may neither overflow nor lose small
tensors), what a single product, a constant plane and a tiny tensor may be off by, and the 16-bit filter gradient of
a few row and column tiles (on single SMs; on pairs: test_gpu_pair_forms.py)."""
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
# both widths; filter gradients of one to four row tiles and of one to three column tiles
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
# value and less) stay normal numbers: filters of 2^-103, whose low parts are 2^-115 and some octaves less. (Further down: test_fp32_tiny_filters.)
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


# What the split drops of a product: lo * lo, at most 2^-22 of it, and of either lo the bits behind the eleven that TF32 holds, at most 2^-23 each. The sum
# of one product and zeros adds no more than the rounding of the result (the additions of the MMAs are exact). Measured: 4.0e-7.
def test_fp32_single_products(gpu):
    n, ci, co, h, w = 2, 40, 48, 12, 16
    rng = np.random.default_rng(68)
    x = np.zeros((4 * n, ci, h, w), np.float32)
    comp, chan = rng.integers(0, 4, (n, h, w)), rng.integers(0, ci, (n, h, w))
    i, a, b = np.meshgrid(np.arange(n), np.arange(h), np.arange(w), indexing="ij")
    value = rng.normal(size=(n, h, w)).astype(np.float32)
    x[comp * n + i, chan, a, b] = value
    f = normal(69, (4, co, ci, 1, 1), std=0.1)
    y = gpu.run_conv_fwd(x, f, None, (1, 1), (0, 0, 0, 0), "f32", "16p", "tensor").reshape(4, n, co, h, w)
    for d in range(4):
        want = np.abs(value[..., None].astype(np.float64) * f[comp ^ d, :, chan, 0, 0])            # [n, h, w, co]; the signs are the oracle tests'
        got = np.abs(np.moveaxis(y[d], 1, -1))
        assert np.max(np.abs(got / want - 1)) <= 2.0 ** -22 + 2 * 2.0 ** -23 + 2.0 ** -24


# Planes and filters of one value: all errors of the products have one sign, and so have those of the additions, which cut off up to 2^-23 of an accumulator that
# grows linearly over at most 64 MMAs: half of half of 64 * 2^-23 on average, beside 2^-21 for the products. The pairs of values have low parts and
# bf16 roundings of one sign.
@pytest.mark.parametrize("a,b", [(1.00146, 1.00146), (1.0024409, 1.0024409), (1 / 3, 0.7), (1.0004, 1.00487)])
@pytest.mark.parametrize("ci,co,k", [(32, 32, 1), (64, 40, 3), (128, 64, 3)])
def test_fp32_constant_planes(gpu, ci, co, k, a, b):
    n, h, w = 2, 14, 16
    x, f = np.zeros((4 * n, ci, h, w), np.float32), np.zeros((4, co, ci, k, k), np.float32)
    x[:n], f[0] = a, b
    y = gpu.run_conv_fwd(x, f, None, (1, 1), (k // 2,) * 4, "f32", "16p", "tensor")[:n]
    taps = np.outer(*(np.convolve(np.ones(s), np.ones(k), "same") for s in (h, w)))
    want = np.float64(np.float32(a)) * np.float64(np.float32(b)) * ci * taps
    assert np.max(np.abs(y / want - 1)) <= 16 * 2.0 ** -23 + 2.0 ** -21 + 2.0 ** -24


# Filters whose low parts are no longer normal numbers keep them to 2^-136, the last bit of a TF32 number; what is cut off is 2^-136 / sqrt(3) on average (in the
# 2-norm), here of filters of 0.053 * 2^-116.
def test_fp32_tiny_filters(gpu):
    n, ci, co, h, w = 4, 20, 24, 26, 17
    std, ew = (2.0 / (4 * ci * 9)) ** 0.5, -116
    x, f = normal(74, (4 * n, ci, h, w)), normal(75, (4, co, ci, 3, 3), std=std)
    pad = (1, 1, 1, 1)
    y = gpu.run_conv_fwd(x, f, None, (1, 1), pad, "f32", "16p", "tensor").astype(np.float64)
    ys = gpu.run_conv_fwd(x * np.float32(2.0 ** 100), f * np.float32(2.0 ** ew), None, (1, 1), pad, "f32", "16p", "tensor").astype(np.float64)
    assert np.linalg.norm(ys * 2.0 ** -(100 + ew) - y) / np.linalg.norm(y) <= 2.0 ** -136 / (std * 2.0 ** ew)
