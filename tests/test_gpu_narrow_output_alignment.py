"""Narrow layers whose output is 16-byte but not 32-byte aligned: they take tiles of 8 instead of 16 pixels, and only layers whose tiles of 8 fit
shared memory may reach those kernels at all. The shapes are a plain 3x3 layer, which falls back, and the smallest ones of which the tile of
16 fits and the tile of 8 does not."""
import numpy as np
import pytest
import torch

from helpers import normal, rel_err, uniform

pytestmark = pytest.mark.gpu

TOL = 2.0 ** -10      # half a unit in the last place of max|ref|, twice for the sums' own error


def _offset(shape, dtype):
    """A contiguous NaN tensor that starts 16 bytes behind a 32-byte boundary."""
    count = int(np.prod(shape))
    t = torch.full((count + 32,), float("nan"), dtype=dtype, device="cuda")
    at = 8 if t.data_ptr() % 32 == 0 else 16
    v = t[at:at + count].view(shape)
    assert v.data_ptr() % 32 == 16
    return v


# algebra, real-valued input, ci, co, h, w, kh, kw, dilation
@pytest.mark.parametrize("case", [
    ("QUATERNION", False, 16, 16, 24, 32, 3, 3, 1), ("QUATERNION", False, 8, 16, 19, 16, 2, 6, 1), ("QUATERNION", False, 16, 8, 31, 32, 2, 5, 2),
    ("QUATERNION", False, 16, 16, 27, 16, 1, 9, 2), ("COMPLEX", False, 16, 16, 32, 32, 3, 7, 1), ("QUATERNION", True, 16, 8, 32, 32, 5, 8, 1),
    ("QUATERNION", True, 8, 16, 28, 48, 6, 7, 1),
])
def test_output_at_an_odd_multiple_of_16_bytes(oracle, case):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import gpu_util as gpu
    import phoenix_core_b200 as pcb
    algebra, real, ci, co, h, w, kh, kw, dil = case
    n, nc = 3, 4 if algebra == "QUATERNION" else 2
    pad = ((kh - 1) * dil // 2, (kw - 1) * dil // 2, (kh - 1) * dil - (kh - 1) * dil // 2, (kw - 1) * dil - (kw - 1) * dil // 2)
    x = gpu.rounded(uniform(71, ((1 if real else nc) * n, ci, h, w)), "f16")
    f = gpu.rounded(normal(72, (nc, co, ci, kh, kw), std=(2.0 / (nc * ci * kh * kw)) ** 0.5), "f16")
    fwd, bwd = gpu.conv_descriptors(x.shape, f.shape, (1, 1), pad, False, not real, real, pcb.Algebra[algebra], (dil, dil))
    code = getattr(oracle, algebra)
    ref = oracle.conv2d_fwd(x, f, None, (1, 1), (dil, dil), pad, code, oracle.VARIANT_16P, real)
    y = _offset(fwd.getOutputShape(), torch.float16)
    pcb.conv2DFwd(gpu.dev(x, "f16"), gpu.dev(f, "f16"), None, y, fwd, gpu.context("16p"), gpu.ENGINES["tensor"])
    assert rel_err(gpu.host(y), ref) <= TOL
    if real:
        return
    dy = gpu.rounded(normal(73, ref.shape), "f16")
    rdw, rdx = oracle.conv2d_bwd(x, f, dy, (1, 1), (dil, dil), pad, code)
    dw, dx = torch.full(f.shape, float("nan"), dtype=torch.float16, device="cuda"), _offset(x.shape, torch.float16)
    pcb.conv2DBwd(gpu.dev(x, "f16"), gpu.dev(f, "f16"), gpu.dev(dy, "f16"), dw, dx, bwd, gpu.context("16p"), gpu.ENGINES["tensor"])
    assert rel_err(gpu.host(dx), rdx) <= TOL and rel_err(gpu.host(dw), rdw) <= TOL
