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
