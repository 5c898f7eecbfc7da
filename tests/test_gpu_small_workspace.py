"""Calls whose workspace is smaller than what the size query asks for, but large enough for the kernels' smallest layout (channels in
slices of 16, copies that end at the last pixel a tap reads): accepted, the same results, no write beyond the workspace."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

# dtype, n, ci, co, h, w, kh, kw, stride, pad, other fields
LAYERS = {
    "slices_of_16": ("f16", 2, 40, 72, 13, 15, 3, 3, 1, 1, {}),
    "several_blocks": ("bf16", 3, 136, 72, 9, 9, 3, 1, 1, 0, {}),
    "pointwise_odd": ("f16", 2, 35, 40, 15, 15, 1, 1, 1, 0, {}),
    "strided_unpadded": ("f16", 2, 40, 48, 18, 20, 3, 3, 2, 0, {}),
    "pixel_classes": ("bf16", 2, 40, 72, 16, 18, 3, 3, 2, 1, {}),
    "stride_classes": ("f16", 2, 40, 66, 16, 18, 1, 3, 2, 0, {}),
    "channels_last": ("f16", 2, 72, 40, 14, 16, 3, 3, 2, 0, {"data_format": 1}),
    "groups": ("f16", 2, 40, 80, 14, 16, 3, 3, 2, 0, {"groups": 2}),
    "real_valued": ("f16", 2, 40, 33, 18, 20, 3, 3, 2, 0, {"real_valued_input": 1, "require_input_grad": 0}),
    "f32_strided_unpadded": ("f32", 2, 40, 24, 18, 20, 3, 3, 2, 0, {}),
    "f32_large_taps": ("f32", 2, 33, 40, 30, 30, 5, 5, 2, 0, {}),
}
# the sums are cut at other places of the channels: twice half a unit in the last place of the largest result, fp32 as elsewhere
TYPES = {"f32": (0, torch.float32, 1e-5), "f16": (1, torch.float16, 2.0 ** -10), "bf16": (2, torch.bfloat16, 2.0 ** -7)}
GUARD = 1 << 16


@pytest.mark.parametrize("name", sorted(LAYERS))
def test_smallest_workspace(name):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from phoenix_core_b200 import _lib
    L = _lib.lib()
    dtype, n, ci, co, h, w, kh, kw, stride, pad, more = LAYERS[name]
    code, t, tol = TYPES[dtype]
    fields = dict(dtype=code, n=n, ci=ci, co=co, h=h, w=w, kh=kh, kw=kw, stride_h=stride, stride_w=stride, dilation_h=1, dilation_w=1,
                  pad_top=pad, pad_left=pad, pad_bottom=pad, pad_right=pad, groups=1, require_input_grad=1)
    fields.update(more)
    d = _lib.ConvDesc(**fields)
    ho, wo = ctypes.c_int32(), ctypes.c_int32()
    _lib.check(L.pcb_conv2d_output_size(ctypes.byref(d), ctypes.byref(ho), ctypes.byref(wo)))
    gen = torch.Generator(device="cuda").manual_seed(11)

    def normal(count, std):
        return (torch.randn(count, generator=gen, device="cuda") * std).to(t)

    real = fields.get("real_valued_input", 0)
    x = normal((1 if real else 4) * n * ci * fields["groups"] * h * w, 1.0)
    f, dy = normal(4 * co * ci * kh * kw, (1.0 / (4 * ci * kh * kw)) ** 0.5), normal(4 * n * co * ho.value * wo.value, 1.0)
    stream = torch.cuda.current_stream().cuda_stream
    grew = False
    for backward in (False, True):
        need = (L.pcb_qconv2d_bwd_workspace_size if backward else L.pcb_qconv2d_fwd_workspace_size)(ctypes.byref(d))
        ws = torch.zeros(need + GUARD, dtype=torch.uint8, device="cuda")

        def call(size):
            out = [torch.full_like(v, float("nan")) for v in ((f, x) if backward else (dy,))]
            p = [v.data_ptr() for v in (x, f, dy, ws, *out)]
            ws.fill_(0xa5)
            if backward:
                rc = L.pcb_qconv2d_bwd(ctypes.byref(d), p[0], p[1], p[2], p[4], None if real else p[5], p[3], size, stream)
            else:
                rc = L.pcb_qconv2d_fwd(ctypes.byref(d), p[0], p[1], None, p[4], p[3], size, stream)
            if rc == _lib.PCB_OK:
                assert L.pcb_check_device_status(p[3], size, stream) == _lib.PCB_OK
                assert bool((ws[size:] == 0xa5).all()), "a write beyond the workspace"
            return rc, (out[:1] if backward and real else out)

        rc, full = call(need)
        _lib.check(rc)
        low, high = 0, need                              # the smallest size that is accepted (in steps of the scratch's alignment)
        while high - low > 256:
            mid = low + (high - low) // 512 * 256
            if mid == low:
                break
            rc, _ = call(mid)
            assert rc in (_lib.PCB_OK, _lib.PCB_ERR_WORKSPACE)
            low, high = (low, mid) if rc == _lib.PCB_OK else (mid, high)
        grew = grew or high < need
        rc, small = call(high)
        _lib.check(rc)
        for a, b in zip(full, small):
            a, b = a.double(), b.double()
            assert torch.isfinite(b).all() and ((a - b).abs().max() / a.abs().max()).item() <= tol
    assert grew


def test_kept_input_is_not_read_in_another_layout():
    """The forward call keeps its staged input, the backward call has the smaller workspace (and the reverse)."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from phoenix_core_b200 import _lib
    L = _lib.lib()
    d = _lib.ConvDesc(dtype=1, n=2, ci=64, co=40, h=18, w=20, kh=3, kw=3, stride_h=2, stride_w=2, dilation_h=1, dilation_w=1, groups=1,
                      require_input_grad=1)
    gen = torch.Generator(device="cuda").manual_seed(12)
    x, f, dy = ((torch.randn(c, generator=gen, device="cuda") * s).half() for c, s in
                ((4 * 2 * 64 * 18 * 20, 1.0), (4 * 40 * 64 * 9, 0.02), (4 * 2 * 40 * 8 * 9, 1.0)))
    fneed, bneed = L.pcb_qconv2d_fwd_workspace_size(ctypes.byref(d)), L.pcb_qconv2d_bwd_workspace_size(ctypes.byref(d))
    stream = torch.cuda.current_stream().cuda_stream
    results = []
    for fsize, bsize in ((fneed, bneed), (fneed, bneed - 256), (fneed - 256, bneed)):
        fws, bws = (torch.zeros(s, dtype=torch.uint8, device="cuda") for s in (fneed, bneed))
        y, dw, dx = (torch.full_like(v, float("nan")) for v in (dy, f, x))
        p = [v.data_ptr() for v in (x, f, dy, y, dw, dx, fws, bws)]
        _lib.check(L.pcb_qconv2d_fwd(ctypes.byref(d), p[0], p[1], None, p[3], p[6], fsize, stream))
        _lib.check(L.pcb_qconv2d_bwd_kept(ctypes.byref(d), p[0], p[1], p[2], p[4], p[5], p[7], bsize, p[6], fsize, stream))
        results.append([v.double() for v in (y, dw, dx)])
    for other in results[1:]:
        for a, b in zip(results[0], other):
            assert torch.isfinite(b).all() and ((a - b).abs().max() / a.abs().max()).item() <= 2.0 ** -10
