"""Workspaces that start at an odd multiple of 16 bytes, the alignment that the calls ask for: every staging kernel stores in units that it allows."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

TYPES = {"f32": (0, torch.float32, 1e-6), "f16": (1, torch.float16, 2.0 ** -10), "bf16": (2, torch.bfloat16, 2.0 ** -7)}


# blocks of 16, 32 and 64 channels (of 32 in the filter gradient), planes whose pixels are loaded four, two and one at a time, tiny planes, a zero-inserted
# gradient, pointwise layers
@pytest.mark.parametrize("dtype,n,ci,co,h,w,k,stride", [
    ("f32", 2, 16, 24, 12, 14, 3, 1), ("f32", 3, 32, 40, 11, 10, 3, 1), ("f32", 2, 72, 64, 9, 7, 3, 1), ("f32", 5, 40, 33, 3, 4, 1, 1), ("f32", 2, 20, 36, 14, 16, 3, 2),
    ("f32", 2, 48, 40, 16, 18, 1, 1), ("f16", 2, 40, 72, 13, 15, 3, 1), ("f16", 2, 12, 16, 24, 32, 3, 1), ("bf16", 3, 128, 128, 14, 14, 1, 1), ("f16", 2, 128, 256, 16, 16, 1, 1),
])
def test_workspace_at_an_odd_multiple_of_16_bytes(dtype, n, ci, co, h, w, k, stride):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from phoenix_core_b200 import _lib
    L = _lib.lib()
    code, t, tol = TYPES[dtype]
    pad = k // 2
    d = _lib.ConvDesc(dtype=code, n=n, ci=ci, co=co, h=h, w=w, kh=k, kw=k, stride_h=stride, stride_w=stride, dilation_h=1, dilation_w=1,
                      pad_top=pad, pad_left=pad, pad_bottom=pad, pad_right=pad, groups=1, require_input_grad=1)
    ho, wo = ctypes.c_int32(), ctypes.c_int32()
    _lib.check(L.pcb_conv2d_output_size(ctypes.byref(d), ctypes.byref(ho), ctypes.byref(wo)))
    gen = torch.Generator(device="cuda").manual_seed(13)
    x, f, dy = ((torch.randn(count, generator=gen, device="cuda") * std).to(t) for count, std in
                ((4 * n * ci * h * w, 1.0), (4 * co * ci * k * k, (1.0 / (4 * ci * k * k)) ** 0.5), (4 * n * co * ho.value * wo.value, 1.0)))
    need = max(L.pcb_qconv2d_fwd_workspace_size(ctypes.byref(d)), L.pcb_qconv2d_bwd_workspace_size(ctypes.byref(d)))
    ws = torch.zeros(need + 64, dtype=torch.uint8, device="cuda")
    assert ws.data_ptr() % 32 == 0
    stream = torch.cuda.current_stream().cuda_stream
    results = []
    for offset in (0, 16):
        y, dw, dx = (torch.full_like(v, float("nan")) for v in (dy, f, x))
        at = ws.data_ptr() + offset
        _lib.check(L.pcb_qconv2d_fwd(ctypes.byref(d), x.data_ptr(), f.data_ptr(), None, y.data_ptr(), at, need, stream))
        _lib.check(L.pcb_qconv2d_bwd(ctypes.byref(d), x.data_ptr(), f.data_ptr(), dy.data_ptr(), dw.data_ptr(), dx.data_ptr(), at, need, stream))
        results.append((y, dw, dx))
    # the same sums, those of split reductions in any order
    for a, b, what in zip(*results, ("y", "dw", "dx")):
        a, b = a.double(), b.double()
        assert torch.isfinite(b).all() and float((a - b).abs().max() / a.abs().max()) <= tol, what
