"""Filter gradient of narrow 16-bit layers whose taps do not fit the tensor memory at once: the groups the taps are dealt into
must each stay within the 512 accumulator columns. Filters of 3 columns fold into 192 columns per row for quaternions (two rows per
group, although five rows over two groups would be three), 96 for two components; GA(3,0,0) and unfolded filters have one tap each."""
import numpy as np
import pytest
import torch

from helpers import normal, rel_err, uniform

pytestmark = pytest.mark.gpu

TOL = {"f16": 2.0 ** -10, "bf16": 2.0 ** -7}      # half a unit in the last place of max|ref|, twice for the sums' own error


@pytest.mark.parametrize("taps,ci,co,h,w,dtype", [((5, 3), 8, 31, 9, 9, "bf16"), ((7, 3), 1, 26, 13, 14, "bf16"), ((5, 3), 16, 16, 20, 24, "f16"),
                                                  ((7, 3), 16, 16, 33, 12, "f16"), ((4, 3), 5, 7, 11, 10, "f16"), ((5, 2), 8, 8, 12, 9, "f16"),
                                                  ((7, 1), 8, 8, 12, 9, "f16"), ((9, 3), 4, 4, 16, 16, "f16")])
def test_tap_groups(oracle, taps, ci, co, h, w, dtype):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import gpu_util as gpu
    kh, kw = taps
    pad = (kh // 2, kw // 2, (kh - 1) // 2, (kw - 1) // 2)
    x = gpu.rounded(uniform(31, (4 * 2, ci, h, w)), dtype)
    f = gpu.rounded(normal(32, (4, co, ci, kh, kw), std=(2.0 / (4 * ci * kh * kw)) ** 0.5), dtype)
    y = oracle.conv2d_fwd(x, f, None, (1, 1), (1, 1), pad)
    dy = gpu.rounded(normal(33, y.shape), dtype)
    rdw, rdx = oracle.conv2d_bwd(x, f, dy, (1, 1), (1, 1), pad)
    dw, dx = gpu.run_conv_bwd(x, f, dy, (1, 1), pad, dtype, "16p", "tensor", True)
    assert np.all(np.isfinite(dw)) and rel_err(dw, rdw) <= TOL[dtype]
    assert np.all(np.isfinite(dx)) and rel_err(dx, rdx) <= TOL[dtype]


@pytest.mark.parametrize("taps,stride,ci,dtype", [((11, 3), 2, 3, "f16"), ((12, 4), 2, 4, "bf16"), ((12, 4), 2, 1, "f16"), ((6, 2), 1, 16, "f16"), ((7, 7), 2, 3, "f16")])
def test_rows_folded_by_halves(oracle, taps, stride, ci, dtype):
    """Real-valued input: the filter rows share an MMA too, three of six here, two of four for the 7 x 7 stem."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import gpu_util as gpu
    kh, kw = taps
    n, h, w = 2, 34, 38
    pad = ((kh - 1) // 2, (kw - 1) // 2, kh // 2, kw // 2)
    x = gpu.rounded(uniform(34, (n, ci, h, w)), dtype)
    f = gpu.rounded(normal(35, (4, 16, ci, kh, kw), std=(2.0 / (ci * kh * kw)) ** 0.5), dtype)
    x4 = np.concatenate([x, np.zeros((3 * n, ci, h, w), np.float32)])            # the quaternions with zero imaginary parts
    dy = gpu.rounded(normal(36, oracle.conv2d_fwd(x4, f, None, (stride, stride), (1, 1), pad).shape), dtype)
    rdw, _ = oracle.conv2d_bwd(x4, f, dy, (stride, stride), (1, 1), pad)
    _, desc = gpu.conv_descriptors(x.shape, f.shape, (stride, stride), pad, False, False, True)
    out = torch.full(f.shape, float("nan"), dtype=gpu.TORCH_DTYPES[dtype], device="cuda")
    gpu.pcb.conv2DBwd(gpu.dev(x, dtype), gpu.dev(f, dtype), gpu.dev(dy, dtype), out, None, desc, gpu.context("16p"), gpu.ENGINES["tensor"])
    dw = gpu.host(out)
    assert np.all(np.isfinite(dw)) and rel_err(dw, rdw) <= TOL[dtype]
