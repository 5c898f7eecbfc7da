"""Narrow 16-bit layers (at most 16 channels): forward and backward-data in tiles of 16 pixels where image rows are whole runs of 16, and the
filter gradient that reads dy in place where the input gradient is not asked for. Heights and widths around whole tiles, 1 to 128 rows of
(component, channel), filters whose taps fold completely, by halves and not at all, strided stems."""
import numpy as np
import pytest
import torch

from helpers import normal, rel_err, uniform

pytestmark = pytest.mark.gpu

TOL = {"f16": 2.0 ** -10, "bf16": 2.0 ** -7}      # half a unit in the last place of max|ref|, twice for the sums' own error


@pytest.fixture(scope="module")
def gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import gpu_util
    return gpu_util


# n, ci, co, h, w, kh, kw
@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("case", [(2, 16, 16, 17, 16, 3, 3), (1, 16, 32, 33, 48, 3, 3), (3, 5, 7, 9, 32, 1, 3), (1, 8, 2, 40, 64, 5, 5), (2, 16, 30, 8, 16, 3, 1),
                                  (2, 12, 24, 31, 112, 2, 2), (1, 16, 16, 15, 40, 3, 3)])
def test_quaternion_layers(gpu, oracle, dtype, case):
    n, ci, co, h, w, kh, kw = case
    pad = (kh // 2, kw // 2, (kh - 1) // 2, (kw - 1) // 2)
    x = gpu.rounded(uniform(41, (4 * n, ci, h, w)), dtype)
    f = gpu.rounded(normal(42, (4, co, ci, kh, kw), std=(2.0 / (4 * ci * kh * kw)) ** 0.5), dtype)
    b = gpu.rounded(uniform(43, (4, co)), dtype)
    ref = oracle.conv2d_fwd(x, f, b, (1, 1), (1, 1), pad)
    y = gpu.run_conv_fwd(x, f, b, (1, 1), pad, dtype, "16p", "tensor")
    assert np.all(np.isfinite(y)) and rel_err(y, ref) <= TOL[dtype]
    dy = gpu.rounded(normal(44, ref.shape), dtype)
    rdw, rdx = oracle.conv2d_bwd(x, f, dy, (1, 1), (1, 1), pad)
    dw, dx = gpu.run_conv_bwd(x, f, dy, (1, 1), pad, dtype, "16p", "tensor", True)
    alone, _ = gpu.run_conv_bwd(x, f, dy, (1, 1), pad, dtype, "16p", "tensor", False)
    for got, want in ((dw, rdw), (dx, rdx), (alone, rdw)):
        assert np.all(np.isfinite(got)) and rel_err(got, want) <= TOL[dtype]


# real-valued inputs; ci, co, h, w, k, stride
@pytest.mark.parametrize("case", [(3, 16, 64, 64, 7, 2), (3, 16, 50, 80, 7, 2), (3, 8, 61, 128, 5, 2), (1, 32, 36, 64, 3, 2), (4, 16, 34, 112, 7, 2), (12, 16, 19, 32, 3, 1),
                                  (16, 6, 12, 56, 4, 1)])
def test_real_valued_input(gpu, oracle, case):
    ci, co, h, w, k, stride = case
    n, dtype = 2, "f16"
    ho, wo = -(-h // stride), -(-w // stride)
    ph, pw = max((ho - 1) * stride + k - h, 0), max((wo - 1) * stride + k - w, 0)
    pad = (ph // 2, pw // 2, ph - ph // 2, pw - pw // 2)
    x = gpu.rounded(uniform(45, (n, ci, h, w)), dtype)
    f = gpu.rounded(normal(46, (4, co, ci, k, k), std=(2.0 / (ci * k * k)) ** 0.5), dtype)
    x4 = np.concatenate([x, np.zeros((3 * n, ci, h, w), np.float32)])            # the quaternions with zero imaginary parts
    ref = oracle.conv2d_fwd(x4, f, None, (stride, stride), (1, 1), pad)
    y = gpu.run_conv_fwd(x, f, None, (stride, stride), pad, dtype, "16p", "tensor", True)
    assert np.all(np.isfinite(y)) and rel_err(y, ref) <= TOL[dtype]
    dy = gpu.rounded(normal(47, ref.shape), dtype)
    rdw, _ = oracle.conv2d_bwd(x4, f, dy, (stride, stride), (1, 1), pad)
    _, desc = gpu.conv_descriptors(x.shape, f.shape, (stride, stride), pad, False, False, True)
    out = torch.full(f.shape, float("nan"), dtype=gpu.TORCH_DTYPES[dtype], device="cuda")
    gpu.pcb.conv2DBwd(gpu.dev(x, dtype), gpu.dev(f, dtype), gpu.dev(dy, dtype), out, None, desc, gpu.context("16p"), gpu.ENGINES["tensor"])
    dw = gpu.host(out)
    assert np.all(np.isfinite(dw)) and rel_err(dw, rdw) <= TOL[dtype]
