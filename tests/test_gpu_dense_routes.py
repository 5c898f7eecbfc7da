"""Which dense calls run on the kernels that read the caller's tensors as they are (they touch only the status block of the workspace) and
which on the staged, persistent ones (they fill the scratch behind it)."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

TYPES = {"f32": (0, torch.float32, 1e-5), "f16": (1, torch.float16, 2.0 ** -10)}
HEADER = 256


@pytest.fixture(scope="module")
def lib():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from phoenix_core_b200 import _lib
    return _lib


def _run(lib, dtype, batch, ci, co, backward, need_dx=True):
    """(results, whether the scratch was written)"""
    L = lib.lib()
    code, t, _ = TYPES[dtype]
    d = lib.DenseDesc(dtype=code, batch=batch, in_features=ci, out_features=co, require_input_grad=int(need_dx))
    gen = torch.Generator(device="cuda").manual_seed(3)
    x, w, dy = ((torch.randn(shape, generator=gen, device="cuda") * std).to(t)
                for shape, std in (((4 * batch, ci), 1.0), ((4, ci, co), (1.0 / (4 * ci)) ** 0.5), ((4 * batch, co), 1.0)))
    need = L.pcb_qdense_bwd_workspace_size(ctypes.byref(d)) if backward else L.pcb_qdense_fwd_workspace_size(ctypes.byref(d))
    ws = torch.full((need,), 0xA5, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    if backward:
        dw, dx = torch.empty_like(w), torch.empty_like(x)
        lib.check(L.pcb_qdense_bwd(ctypes.byref(d), x.data_ptr(), w.data_ptr(), dy.data_ptr(), dw.data_ptr(), dx.data_ptr() if need_dx else None,
                                   ws.data_ptr(), need, stream))
        out = [dw, dx] if need_dx else [dw]
    else:
        y = torch.empty_like(dy)
        lib.check(L.pcb_qdense_fwd(ctypes.byref(d), x.data_ptr(), w.data_ptr(), None, y.data_ptr(), ws.data_ptr(), need, stream))
        out = [y]
    assert L.pcb_check_device_status(ws.data_ptr(), need, stream) == lib.PCB_OK
    return out, bool((ws[HEADER:] != 0xA5).any())


@pytest.mark.parametrize("backward", [False, True])
@pytest.mark.parametrize("dtype", ["f32", "f16"])
@pytest.mark.parametrize("batch,ci,co,fits", [(32, 64, 64, True), (1024, 512, 1280, False)])
def test_sm_margin(lib, dtype, backward, batch, ci, co, fits):
    """With a margin, layers of more CTAs than the SMs that are left run on the kernels that size their grids for it."""
    want, staged = _run(lib, dtype, batch, ci, co, backward)
    assert not staged
    try:
        lib.check(lib.lib().pcb_set_sm_margin(8))
        got, staged = _run(lib, dtype, batch, ci, co, backward)
    finally:
        lib.check(lib.lib().pcb_set_sm_margin(0))
    assert staged == (not fits)
    for a, b in zip(got, want):
        assert ((a.double() - b.double()).abs().max() / b.double().abs().max()).item() <= TYPES[dtype][2]


# sizes on both sides of the lines between the two kernel families: dtype, batch, ci, co, and whether (y, dw and dx, dw alone) are staged
@pytest.mark.parametrize("dtype,batch,ci,co,staged", [
    ("f16", 1024, 511, 333, (False, False, False)), ("f16", 4096, 511, 333, (True, False, True)), ("f16", 2048, 1001, 999, (True, True, False)),
    ("f16", 4096, 1024, 511, (True, True, True)), ("f16", 8192, 768, 1024, (True, True, False)), ("f16", 4096, 2048, 1024, (False, True, False)),
    ("f16", 16384, 512, 1024, (True, True, True)), ("f16", 16384, 256, 256, (False, False, False)),
    ("f32", 1024, 512, 512, (False, False, False)), ("f32", 1536, 768, 768, (False, True, True)), ("f32", 1024, 611, 900, (True, False, True)), ("f32", 1024, 768, 701, (False, False, True)),
    ("f32", 768, 512, 512, (False, False, False)), ("f32", 2048, 2048, 512, (True, True, True))])
def test_large_layers(lib, dtype, batch, ci, co, staged):
    t, tol = TYPES[dtype][1:]
    gen = torch.Generator(device="cuda").manual_seed(3)                      # the tensors that _run makes
    x, w, dy = ((torch.randn(shape, generator=gen, device="cuda") * std).to(t)
                for shape, std in (((4 * batch, ci), 1.0), ((4, ci, co), (1.0 / (4 * ci)) ** 0.5), ((4 * batch, co), 1.0)))
    # y = x (Hamilton product) w: component l of x times component l ^ d of w goes into component d of y, with these negative
    negative = {(1, 0), (1, 2), (2, 0), (2, 3), (3, 0), (3, 1)}
    block = torch.cat([torch.cat([(-1.0 if (l, d) in negative else 1.0) * w[l ^ d].double() for d in range(4)], dim=1) for l in range(4)], dim=0)

    def join(v):
        return v.view(4, batch, -1).transpose(0, 1).reshape(batch, -1).double()

    def split(v, c):
        return v.view(batch, 4, c).transpose(0, 1).reshape(4 * batch, c)

    want_y = split(join(x) @ block, co)
    want_dx = split(join(dy) @ block.t(), ci)
    g = join(x).t() @ join(dy)
    want_dw = torch.zeros(4, ci, co, dtype=torch.float64, device="cuda")
    for l in range(4):
        for d in range(4):
            want_dw[l ^ d] += (-1.0 if (l, d) in negative else 1.0) * g[l * ci:(l + 1) * ci, d * co:(d + 1) * co]
    calls = ((False, True, (want_y,)), (True, True, (want_dw, want_dx)), (True, False, (want_dw,)))
    for (backward, need_dx, want), expected in zip(calls, staged):
        got, was_staged = _run(lib, dtype, batch, ci, co, backward, need_dx)
        assert was_staged == expected, (backward, need_dx)
        for a, b in zip(got, want):
            assert ((a.double() - b).abs().max() / b.abs().max()).item() <= tol
