"""The general kernels and filter gradients on pairs of SMs in every form that a layer can ask for: halo tiles, plain tiles and the strided
backward-data form; channels-last tensors read in place and copied, stored in blocks of 32 channels and element by element; grouped layers, dilation, other
algebras, a kept copy of x, an SM margin, fp32. The layers lie above the line below which single SMs are taken, and every test asks the profiler which kernels
ran. The reference is the fp32 kernel of the CUDA cores on the same rounded inputs."""
import re

import pytest
import torch

pytestmark = pytest.mark.gpu

# half a unit in the last place of max|ref|, twice for the sums' own error; fp32 as elsewhere
TOL = {"f32": 1e-5, "f16": 2.0 ** -10, "bf16": 2.0 ** -7}
HALO, PLAIN, DUAL = r"qconv_general_tc_kernel<32, true, false, true>", r"qconv_general_tc_kernel<\d+, false, false, true>", r"qconv_general_tc_kernel<\d+, false, true, true>"
FILTER = r"qconv_filter_general_tc_kernel<true>"
F32, F32_HALO, F32_FILTER = r"qconv_general_tf32_kernel<\w+, false, true>", r"qconv_general_tf32_kernel<\w+, true, true>", r"qconv_filter_tf32_kernel<true>"


def _kernels(call):
    """Names of the kernels that a call launches."""
    from torch.profiler import ProfilerActivity, profile
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        call()
        torch.cuda.synchronize()
    return [e.key for e in p.key_averages() if "pcb::" in e.key]


def _case(dtype, n, ci, co, h, w, k, stride=1, nhwc=False, groups=1, dil=1, algebra="QUATERNION", keep=False, margin=0, fwd=HALO, data=None, grad=FILTER):
    return dict(locals())


CASES = [
    _case("f16", 16, 64, 64, 30, 24, 3, nhwc=True),                                              # in place, blocks of 32 channels
    _case("bf16", 14, 64, 32, 57, 30, 3, nhwc=True, data=HALO, grad="", fwd=""),                 # one row tile forward, two backward
    _case("f16", 30, 128, 128, 28, 28, 3, 2, nhwc=True, fwd=PLAIN, data=DUAL),
    _case("bf16", 30, 128, 128, 14, 14, 3, nhwc=True, fwd=PLAIN),
    _case("f16", 24, 40, 56, 31, 30, 3, nhwc=True),                                              # copied, stored element by element
    _case("f16", 30, 40, 56, 40, 30, 3, 2, nhwc=True, fwd=PLAIN, data=DUAL),
    _case("bf16", 90, 56, 40, 31, 29, 1, nhwc=True, fwd=PLAIN, data=PLAIN, grad=""),
    _case("f16", 16, 128, 128, 30, 24, 3, groups=2),
    _case("bf16", 60, 96, 112, 30, 28, 3, 2, groups=2, fwd=PLAIN, data=DUAL, grad=""),
    _case("f16", 16, 64, 64, 28, 30, 3, dil=2),
    _case("f16", 16, 64, 64, 28, 30, 3, nhwc=True, dil=2),
    _case("f16", 40, 64, 128, 30, 30, 3, algebra="COMPLEX", data="", grad=""),                   # (backward-data: one row tile)
    _case("bf16", 18, 32, 32, 30, 24, 3, algebra="GA_300"),
    _case("f16", 16, 64, 64, 30, 24, 3, keep=True),
    _case("bf16", 24, 64, 128, 28, 28, 3, 2, keep=True, fwd=PLAIN, data=DUAL),
    _case("f16", 16, 64, 64, 30, 24, 3, nhwc=True, margin=3),
    _case("f16", 24, 64, 128, 28, 28, 3, 2, margin=5, fwd=PLAIN, data=DUAL),
    _case("f16", 14, 64, 64, 45, 33, 3, margin=64),
    _case("f32", 64, 128, 64, 28, 28, 3, fwd=F32_HALO, data=F32_HALO, grad=F32_FILTER),
    _case("f32", 40, 128, 64, 20, 21, 3, 2, fwd=F32, data="", grad=F32_FILTER),
    _case("f32", 60, 256, 256, 14, 14, 1, margin=4, fwd=F32, data=F32, grad=""),
]


@pytest.mark.parametrize("c", CASES, ids=lambda c: "-".join(str(v) for v in list(c.values())[:12]))
def test_pair_forms(c):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import gpu_util as gpu
    import phoenix_core_b200 as pcb
    from phoenix_core_b200 import ops
    alg = pcb.Algebra[c["algebra"]]
    comps = {"COMPLEX": 2, "QUATERNION": 4, "GA_300": 8}[c["algebra"]]
    n, ci, co, h, w, k, g, dtype = c["n"], c["ci"], c["co"], c["h"], c["w"], c["k"], c["groups"], c["dtype"]
    xs = (comps * n, h, w, ci) if c["nhwc"] else (comps * n, ci, h, w)
    ws = (comps, co, k, k, ci // g) if c["nhwc"] else (comps, co, ci // g, k, k)
    args = (xs, ws, c["stride"], c["dil"], pcb.Padding.SAME, (), g, alg, pcb.DataFormat.NHWC if c["nhwc"] else pcb.DataFormat.NCHW,
            pcb.FilterLayout.OHWI if c["nhwc"] else pcb.FilterLayout.OIHW)
    fwd, bwd = pcb.Conv2DFwdDescriptor(*args, True), pcb.Conv2DBwdDescriptor(*args, True)
    gen = torch.Generator(device="cuda").manual_seed(91)
    t = gpu.TORCH_DTYPES[dtype]
    x, f, b, dy = (torch.randn(s, generator=gen, device="cuda").mul_(std).to(t) for s, std in
                   ((xs, 1.0), (ws, (2.0 / (comps * ci // g * k * k)) ** 0.5), ((comps, co), 0.1), (fwd.getOutputShape(), 1.0)))
    ctx, simt = gpu.context("16p"), gpu.ENGINES["simt"]

    def outputs(like):
        return [torch.full(s, float("nan"), dtype=like, device="cuda") for s in (fwd.getOutputShape(), ws, xs)]

    y, dw, dx = outputs(t)
    kept = pcb.KeptInput() if c["keep"] else None
    engine = gpu.ENGINES["auto" if c["keep"] else "tensor"]
    ops.setSmMargin(c["margin"])
    try:
        ran = _kernels(lambda: pcb.conv2DFwd(x, f, b, y, fwd, ctx, engine, keep=kept))
        if c["keep"]:
            assert kept.workspace is not None
        ran_b = _kernels(lambda: pcb.conv2DBwd(x, f, dy, dw, dx, bwd, ctx, engine, kept=kept))
    finally:
        ops.setSmMargin(0)
    if ran and ran_b:                                    # (no names where the profiler is not available)
        for names, wanted in ((ran, c["fwd"]), (ran_b, c["fwd"] if c["data"] is None else c["data"]), (ran_b, c["grad"])):
            assert any(re.search(wanted, name) for name in names), (wanted, [name.split("(CUtensor")[0][-60:] for name in names])
    ry, rdw, rdx = outputs(torch.float32)
    x32, f32, b32, dy32 = (v.float() for v in (x, f, b, dy))
    pcb.conv2DFwd(x32, f32, b32, ry, fwd, ctx, simt)
    pcb.conv2DBwd(x32, f32, dy32, rdw, rdx, bwd, ctx, simt)
    for got, want, what in ((y, ry, "y"), (dx, rdx, "dx"), (dw, rdw, "dw")):
        assert torch.isfinite(got).all(), what
        err = float((got.double() - want.double()).abs().max() / want.double().abs().max())
        assert err <= TOL[dtype], (what, err)
