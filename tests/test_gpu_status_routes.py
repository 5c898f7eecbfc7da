"""Every kernel family behind the convolution calls, given a workspace whose status word holds an old report: the word is reset in front
of the first kernel that waits (a call that leaves it owing is an error), the results are those of a clean workspace."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

ROUTES = {
    # name: dtype, n, ci, co, h, w, kh, kw, stride, other fields
    "pointwise_pair": ("f16", 150, 64, 256, 8, 8, 1, 1, 1, {}),
    "pointwise": ("bf16", 3, 96, 128, 16, 8, 1, 1, 1, {}),
    "pointwise_few_channels": ("f16", 3, 16, 24, 16, 8, 1, 1, 1, {}),
    "pointwise_8_products": ("f16", 2, 64, 64, 16, 16, 1, 1, 1, {"variant": 1, "engine": 2}),
    "strided_pointwise": ("f16", 3, 64, 96, 16, 16, 1, 1, 2, {}),
    "strided_pointwise_f32": ("f32", 3, 24, 32, 16, 16, 1, 1, 2, {}),
    "narrow": ("f16", 2, 16, 16, 20, 20, 3, 3, 1, {}),
    "narrow_strided": ("f16", 2, 4, 16, 32, 32, 3, 3, 2, {}),
    "general": ("f16", 2, 48, 40, 13, 15, 3, 3, 1, {}),
    "general_dilated": ("bf16", 2, 64, 64, 19, 17, 3, 3, 1, {"dilation_h": 2, "dilation_w": 2}),
    "pixel_classes": ("f16", 2, 64, 96, 16, 18, 3, 3, 2, {}),
    "stride_classes_one_row": ("f16", 2, 136, 64, 16, 18, 1, 3, 2, {}),
    "stride_classes_f32": ("f32", 2, 128, 32, 16, 18, 3, 3, 2, {}),
    "f32": ("f32", 2, 40, 24, 13, 15, 3, 3, 1, {}),
    "f32_cut_reduction": ("f32", 1, 96, 32, 8, 8, 3, 3, 1, {}),
    "channels_last": ("f16", 2, 32, 48, 14, 14, 3, 3, 1, {"data_format": 1, "filter_layout": 1}),
    "channels_last_strided": ("f16", 2, 40, 48, 14, 14, 3, 3, 2, {"data_format": 1, "filter_layout": 2}),
    "groups": ("f16", 2, 24, 64, 14, 14, 3, 3, 1, {"groups": 2}),
    "cuda_cores": ("f32", 2, 8, 8, 9, 9, 3, 3, 1, {"engine": 1}),
}
TYPES = {"f32": (0, torch.float32, 1e-5), "f16": (1, torch.float16, 2.0 ** -10), "bf16": (2, torch.bfloat16, 2.0 ** -7)}


@pytest.mark.parametrize("name", sorted(ROUTES))
def test_old_report_is_cleared_first(name):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from phoenix_core_b200 import _lib
    L = _lib.lib()
    dtype, n, ci, co, h, w, kh, kw, stride, more = ROUTES[name]
    code, t, tol = TYPES[dtype]
    fields = dict(dtype=code, n=n, ci=ci, co=co, h=h, w=w, kh=kh, kw=kw, stride_h=stride, stride_w=stride, dilation_h=1, dilation_w=1,
                  groups=1, require_input_grad=1)
    fields.update(more)
    dil, groups = fields["dilation_h"], fields["groups"]
    fields["pad_top"] = fields["pad_bottom"] = kh // 2 * dil
    fields["pad_left"] = fields["pad_right"] = kw // 2 * dil
    d = _lib.ConvDesc(**fields)
    ho, wo = ctypes.c_int32(), ctypes.c_int32()
    _lib.check(L.pcb_conv2d_output_size(ctypes.byref(d), ctypes.byref(ho), ctypes.byref(wo)))
    gen = torch.Generator(device="cuda").manual_seed(7)

    def normal(count, std):
        return (torch.randn(count, generator=gen, device="cuda") * std).to(t)

    x, f, dy = normal(4 * n * ci * groups * h * w, 1.0), normal(4 * co * ci * kh * kw, (1.0 / (4 * ci * kh * kw)) ** 0.5), normal(4 * n * co * ho.value * wo.value, 1.0)
    need = max(L.pcb_qconv2d_fwd_workspace_size(ctypes.byref(d)), L.pcb_qconv2d_bwd_workspace_size(ctypes.byref(d)))
    ws = torch.zeros(need, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    results = []
    for word in (0, 0x7fffffff):
        y, dw, dx = (torch.full_like(v, float("nan")) for v in (dy, f, x))
        ptr = [v.data_ptr() for v in (x, f, dy, y, dw, dx, ws)]
        calls = [lambda: L.pcb_qconv2d_fwd(ctypes.byref(d), ptr[0], ptr[1], None, ptr[3], ptr[6], need, stream),
                 lambda: L.pcb_qconv2d_bwd(ctypes.byref(d), ptr[0], ptr[1], ptr[2], ptr[4], ptr[5], ptr[6], need, stream),
                 lambda: L.pcb_qconv2d_bwd_data(ctypes.byref(d), ptr[1], ptr[2], ptr[5], ptr[6], need, stream),
                 lambda: L.pcb_qconv2d_bwd_filter(ctypes.byref(d), ptr[0], ptr[2], ptr[4], ptr[6], need, stream)]
        for call in calls:
            ws[:4].view(torch.int32).fill_(word)
            _lib.check(call())
            assert L.pcb_check_device_status(ptr[6], need, stream) == _lib.PCB_OK
        results.append((y, dw, dx))
    for clean, old in zip(*results):
        clean, old = clean.double(), old.double()
        assert torch.isfinite(old).all()
        assert ((clean - old).abs().max() / clean.abs().max()).item() <= tol
