"""Host threads that call the C ABI at the same time, each on its own stream and workspace, with layers of one kernel that need different
amounts of shared memory (image rows that are and are not 16-byte aligned): no call may fail or change its result."""
import ctypes
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu

TYPES = {"f32": (0, torch.float32, 1e-5), "f16": (1, torch.float16, 2.0 ** -10)}
# channels, and the widths of the two layers
LAYERS = {"fp32": ("f32", 16, 32, 37), "general": ("f16", 48, 16, 13), "narrow": ("f16", 16, 32, 19), "general_wide": ("f16", 40, 64, 45)}


@pytest.mark.parametrize("name", sorted(LAYERS))
def test_two_threads(name):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from phoenix_core_b200 import _lib
    L = _lib.lib()
    dtype, c, *widths = LAYERS[name]
    code, t, tol = TYPES[dtype]
    n, h = 2, 24
    problems, failures = [], []
    for i, w in enumerate(widths):
        d = _lib.ConvDesc(dtype=code, n=n, ci=c, co=c, h=h, w=w, kh=3, kw=3, stride_h=1, stride_w=1, dilation_h=1, dilation_w=1, pad_top=1, pad_left=1,
                          pad_bottom=1, pad_right=1, groups=1, require_input_grad=1)
        gen = torch.Generator(device="cuda").manual_seed(i)
        x = torch.randn(4 * n * c * h * w, generator=gen, device="cuda").to(t)
        f = (torch.randn(4 * c * c * 9, generator=gen, device="cuda") * (1.0 / (36 * c)) ** 0.5).to(t)
        need = L.pcb_qconv2d_fwd_workspace_size(ctypes.byref(d))
        p = {"d": d, "x": x, "f": f, "y": torch.empty_like(x), "ws": torch.zeros(need, dtype=torch.uint8, device="cuda"), "need": need,
             "stream": torch.cuda.Stream()}
        torch.cuda.synchronize()
        _lib.check(_forward(L, p))
        torch.cuda.synchronize()
        p["want"] = p["y"].clone()
        problems.append(p)
    torch.cuda.synchronize()
    start = threading.Barrier(len(problems))

    def work(p):
        torch.cuda.set_device(0)
        start.wait()
        for _ in range(400):
            status = _forward(L, p)
            if status != 0:
                failures.append((status, L.pcb_last_error_message()))
                return

    threads = [threading.Thread(target=work, args=(p,)) for p in problems]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    torch.cuda.synchronize()
    assert not failures, failures[0]
    for p in problems:
        got, want = p["y"].double(), p["want"].double()
        assert ((got - want).abs().max() / want.abs().max()).item() <= tol


def _forward(L, p):
    return L.pcb_qconv2d_fwd(ctypes.byref(p["d"]), p["x"].data_ptr(), p["f"].data_ptr(), None, p["y"].data_ptr(), p["ws"].data_ptr(), p["need"],
                             p["stream"].cuda_stream)
