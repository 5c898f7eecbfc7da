"""fp32 convolutions on the tensor cores at the sizes where the staging transposition and the row epilogue end: planes of 4k, 2k and
odd pixels, image rows of every alignment, channels around the 16- and 32-channel blocks, a reduction cut over several CTAs (whose
partial sums meet in the zeroed output), one and several row tiles."""
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


# n, ci, co, h, w, k, stride, pad
SHAPES = [(2, 17, 40, 9, 13, 3, (1, 1), (1, 1, 1, 1)), (1, 48, 20, 11, 10, 3, (1, 1), (0, 2, 1, 0)), (3, 33, 33, 6, 12, 1, (1, 1), (0, 0, 0, 0)),
          (2, 8, 8, 20, 21, 5, (2, 2), (2, 2, 2, 2)), (1, 64, 48, 8, 8, 3, (1, 1), (1, 1, 1, 1)), (6, 32, 32, 19, 19, 1, (1, 1), (0, 0, 0, 0)),
          (1, 96, 36, 7, 9, 3, (1, 1), (1, 1, 1, 1)), (2, 5, 6, 5, 4, 3, (1, 1), (1, 1, 1, 1)), (2, 24, 16, 3, 5, 3, (1, 1), (1, 1, 1, 1))]


@pytest.mark.parametrize("shape", SHAPES)
def test_fp32_tile_edges(gpu, oracle, shape):
    n, ci, co, h, w, k, stride, pad = shape
    x = uniform(95, (4 * n, ci, h, w))
    f = normal(96, (4, co, ci, k, k), std=(2.0 / (4 * ci * k * k)) ** 0.5)
    b = uniform(97, (4, co))
    ref = oracle.conv2d_fwd(x, f, b, stride, (1, 1), pad)
    y = gpu.run_conv_fwd(x, f, b, stride, pad, "f32", "16p", "tensor")
    dy = normal(98, ref.shape)
    rdw, rdx = oracle.conv2d_bwd(x, f, dy, stride, (1, 1), pad)
    dw, dx = gpu.run_conv_bwd(x, f, dy, stride, pad, "f32", "16p", "tensor", True)
    for got, want, what in ((y, ref, "y"), (dx, rdx, "dx"), (dw, rdw, "dw")):
        assert np.all(np.isfinite(got)), what
        assert rel_err(got, want) <= 1e-5, (what, rel_err(got, want))


# planes of 1 to 15 pixels: staged thread by thread beside the filters, 1 to 40 channels in blocks of 16 and 32, several images
@pytest.mark.parametrize("shape", [(5, 33, 17, 1, 1, 1, 0), (3, 6, 40, 3, 5, 3, 1), (7, 1, 3, 2, 2, 2, 0), (2, 64, 31, 1, 15, 3, 1), (130, 20, 24, 3, 3, 3, 1)])
def test_fp32_tiny_planes(gpu, oracle, shape):
    n, ci, co, h, w, k, p = shape
    pad = (p, p, p, p)
    x = uniform(95, (4 * n, ci, h, w))
    f = normal(96, (4, co, ci, k, k), std=(2.0 / (4 * ci * k * k)) ** 0.5)
    ref = oracle.conv2d_fwd(x, f, None, (1, 1), (1, 1), pad)
    y = gpu.run_conv_fwd(x, f, None, (1, 1), pad, "f32", "16p", "tensor")
    dy = normal(98, ref.shape)
    rdw, rdx = oracle.conv2d_bwd(x, f, dy, (1, 1), (1, 1), pad)
    dw, dx = gpu.run_conv_bwd(x, f, dy, (1, 1), pad, "f32", "16p", "tensor", True)
    for got, want, what in ((y, ref, "y"), (dx, rdx, "dx"), (dw, rdw, "dw")):
        assert np.all(np.isfinite(got)), what
        assert rel_err(got, want) <= 1e-5, (what, rel_err(got, want))


# filter matrices of more than 64 MB, gathered across their storage order by a launch of their own: backward-data of a wide 3x3 layer on
# planes of 16 and more and of fewer pixels, with and without a cut reduction
@pytest.mark.parametrize("n,c,h,w", [(1, 256, 5, 6), (3, 264, 3, 4)])
def test_fp32_large_filter_matrix(gpu, oracle, n, c, h, w):
    pad = (1, 1, 1, 1)
    x = uniform(95, (4 * n, c, h, w))
    f = normal(96, (4, c, c, 3, 3), std=(2.0 / (36 * c)) ** 0.5)
    dy = normal(98, (4 * n, c, h, w))
    rdw, rdx = oracle.conv2d_bwd(x, f, dy, (1, 1), (1, 1), pad)
    dw, dx = gpu.run_conv_bwd(x, f, dy, (1, 1), pad, "f32", "16p", "tensor", True)
    for got, want, what in ((dx, rdx, "dx"), (dw, rdw, "dw")):
        assert np.all(np.isfinite(got)), what
        assert rel_err(got, want) <= 1e-5, (what, rel_err(got, want))
