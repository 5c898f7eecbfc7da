"""General kernels of layers with an even number of 128-row tiles: whole planes in a tile, planes of an odd number of rows, power-of-two boxes, halo
tiles; batches that leave part of a tile empty; odd and even planes; slices of 16, 32 and 64 channels; strides, bias, channels-last. The layers of test_pairs
and test_pairs_channels_last are too small for pairs of SMs and run on single ones; those of test_large_layers take pairs where they have two row tiles.
The other forms on pairs, with a check of which kernel ran: test_gpu_pair_forms.py."""
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


def _same(size, k, s):
    out = -(-size // s)
    total = max((out - 1) * s + k - size, 0)
    return total // 2, total - total // 2


# n, ci, co, h, w, k, stride
@pytest.mark.parametrize("dtype,case", [
    ("bf16", (3, 64, 128, 14, 14, 1, 1)), ("f16", (1, 40, 128, 7, 7, 3, 1)), ("f16", (5, 72, 128, 7, 7, 1, 1)), ("f16", (2, 64, 128, 13, 13, 1, 1)),
    ("bf16", (2, 24, 256, 12, 15, 3, 1)), ("f16", (3, 48, 128, 28, 28, 3, 2)), ("f16", (1, 16, 128, 16, 16, 1, 1)), ("f16", (9, 20, 128, 5, 4, 3, 1)),
    ("f16", (2, 64, 64, 20, 24, 1, 1)), ("bf16", (1, 40, 48, 33, 40, 3, 2)), ("f16", (3, 36, 64, 9, 11, 3, 1)), ("f16", (300, 24, 64, 2, 2, 2, 1)),
    ("f16", (1, 64, 64, 25, 17, 3, 1)), ("bf16", (2, 32, 100, 11, 130, 3, 1)), ("f16", (1, 18, 64, 40, 300, 1, 2)),
])
def test_pairs(gpu, oracle, dtype, case):
    n, ci, co, h, w, k, s = case
    (pt, pb), (pl, pr) = _same(h, k, s), _same(w, k, s)
    pad = (pt, pl, pb, pr)
    x = gpu.rounded(uniform(51, (4 * n, ci, h, w)), dtype)
    f = gpu.rounded(normal(52, (4, co, ci, k, k), std=(2.0 / (4 * ci * k * k)) ** 0.5), dtype)
    b = gpu.rounded(uniform(53, (4, co)), dtype)
    ref = oracle.conv2d_fwd(x, f, b, (s, s), (1, 1), pad)
    y = gpu.run_conv_fwd(x, f, b, (s, s), pad, dtype, "16p", "tensor")
    assert np.all(np.isfinite(y)) and rel_err(y, ref) <= TOL[dtype]
    dy = gpu.rounded(normal(54, ref.shape), dtype)
    rdw, rdx = oracle.conv2d_bwd(x, f, dy, (s, s), (1, 1), pad)
    dw, dx = gpu.run_conv_bwd(x, f, dy, (s, s), pad, dtype, "16p", "tensor", True)
    for got, want, what in ((dx, rdx, "dx"), (dw, rdw, "dw")):
        assert np.all(np.isfinite(got)) and rel_err(got, want) <= TOL[dtype], (what, rel_err(got, want))


@pytest.mark.parametrize("co,h,w", [(64, 26, 24), (96, 9, 10)])
def test_pairs_channels_last(gpu, oracle, co, h, w):
    import phoenix_core_b200 as pcb
    n, ci = 2, 48
    x = gpu.rounded(uniform(55, (4 * n, ci, h, w)), "f16")
    f = gpu.rounded(normal(56, (4, co, ci, 3, 3), std=0.03), "f16")
    ref = oracle.conv2d_fwd(x, f, None, (1, 1), (1, 1), (1, 1, 1, 1))
    xd = torch.from_numpy(x).permute(0, 2, 3, 1).contiguous().half().cuda()
    wd = torch.from_numpy(f).permute(0, 1, 3, 4, 2).contiguous().half().cuda()
    desc = pcb.Conv2DFwdDescriptor(tuple(xd.shape), tuple(wd.shape), 1, 1, pcb.Padding.SAME, (), 1, pcb.Algebra.QUATERNION, pcb.DataFormat.NHWC, pcb.FilterLayout.OHWI, False)
    y = torch.full(desc.getOutputShape(), float("nan"), dtype=torch.float16, device="cuda")
    pcb.conv2DFwd(xd, wd, None, y, desc, gpu.context("16p"), gpu.ENGINES["tensor"])
    assert rel_err(y.float().cpu().permute(0, 3, 1, 2).numpy(), ref) <= TOL["f16"]


# Layers with enough MMAs for pairs, and pointwise layers whose planes are taken as rows of pixels (odd and even planes, planes of less and more
# than a tile, tiles of whole rows and of several images). The reference is the fp32 kernel of the CUDA cores on the same rounded inputs.
@pytest.mark.parametrize("dtype,case", [
    ("bf16", (27, 256, 256, 14, 14, 1, 1)), ("f16", (21, 64, 128, 14, 14, 3, 1)), ("f16", (46, 64, 128, 7, 7, 3, 1)), ("f16", (24, 64, 128, 13, 13, 3, 1)),
    ("f16", (17, 64, 128, 28, 28, 3, 2)), ("bf16", (9, 64, 64, 40, 24, 3, 1)), ("f16", (7, 48, 64, 31, 44, 3, 1)), ("f16", (5, 96, 64, 26, 57, 5, 1)),
    ("f16", (40, 64, 128, 28, 28, 3, 2)), ("f16", (33, 64, 96, 41, 30, 3, 2)), ("bf16", (14, 64, 64, 29, 52, 5, 2)), ("f16", (41, 96, 64, 20, 18, 3, 2)), ("f16", (33, 128, 192, 23, 20, 1, 1)), ("bf16", (7, 128, 192, 61, 51, 1, 1)), ("f16", (80, 128, 128, 5, 9, 3, 1)),
    ("f16", (64, 16, 64, 24, 24, 3, 1)), ("f16", (9, 48, 40, 41, 47, 1, 1)), ("bf16", (50, 24, 56, 12, 11, 1, 1)),
    ("f16", (9, 37, 56, 15, 13, 3, 1)), ("f32", (9, 21, 40, 15, 13, 3, 1)), ("bf16", (9, 42, 64, 15, 13, 1, 1)),
    ("f16", (9, 24, 56, 15, 13, 1, 1)), ("bf16", (41, 64, 256, 14, 14, 1, 1)), ("f16", (1, 256, 64, 9, 9, 1, 1)), ("f16", (31, 256, 128, 18, 18, 1, 1)), ("f16", (11, 16, 64, 9, 7, 1, 1)),
    ("f32", (5, 64, 64, 56, 28, 3, 1)), ("f32", (40, 64, 64, 14, 15, 3, 1)), ("f32", (21, 128, 128, 19, 17, 1, 1)), ("f32", (12, 40, 48, 33, 41, 3, 1)),
    ("f32", (9, 40, 24, 41, 47, 1, 1)), ("f32", (33, 96, 64, 24, 20, 3, 2)), ("f32", (3, 16, 24, 101, 37, 3, 1)), ("f32", (5, 24, 32, 40, 51, 1, 1)),
    ("f32", (10, 24, 30, 47, 47, 3, 1)),
])
def test_large_layers(gpu, dtype, case):
    n, ci, co, h, w, k, s = case
    (pt, pb), (pl, pr) = _same(h, k, s), _same(w, k, s)
    pad = (pt, pl, pb, pr)
    x = gpu.rounded(uniform(57, (4 * n, ci, h, w)), dtype)
    f = gpu.rounded(normal(58, (4, co, ci, k, k), std=(2.0 / (4 * ci * k * k)) ** 0.5), dtype)
    b = gpu.rounded(uniform(59, (4, co)), dtype)
    tol = TOL.get(dtype, 1e-5)
    ref = gpu.run_conv_fwd(x, f, b, (s, s), pad, "f32", "16p", "simt")
    y = gpu.run_conv_fwd(x, f, b, (s, s), pad, dtype, "16p", "tensor")
    assert np.all(np.isfinite(y)) and rel_err(y, ref) <= tol, rel_err(y, ref)
    dy = gpu.rounded(normal(60, ref.shape), dtype)
    rdw, rdx = gpu.run_conv_bwd(x, f, dy, (s, s), pad, "f32", "16p", "simt", True)
    dw, dx = gpu.run_conv_bwd(x, f, dy, (s, s), pad, dtype, "16p", "tensor", True)
    for got, want, what in ((dx, rdx, "dx"), (dw, rdw, "dw")):
        assert np.all(np.isfinite(got)) and rel_err(got, want) <= tol, (what, rel_err(got, want))
