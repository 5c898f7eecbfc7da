"""Results that share memory with operands: dense layers and fp32 convolutions stage their operands before anything is written, and the
strided 16-bit backward pass runs the filter gradient before dx replaces x or reads a copy of dy. Compared with the same call on tensors
that lie apart; the two may differ by the order of their sums and the rounding of the stored results."""
import pytest
import torch

pytestmark = pytest.mark.gpu

TYPES = {"f32": (torch.float32, 1e-5), "f16": (torch.float16, 2.0 ** -10), "bf16": (torch.bfloat16, 2.0 ** -7)}


@pytest.fixture(scope="module")
def pcb():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import phoenix_core_b200
    return phoenix_core_b200


def _normal(seed, shape, dtype, std=1.0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(shape, generator=gen, device="cuda") * std).to(dtype)


def _close(got, want, tol):
    got, want = got.double(), want.double()
    assert torch.isfinite(got).all()
    assert ((got - want).abs().max() / want.abs().max()).item() <= tol


def _inside(shape, at, dtype):
    """A tensor at the head of a buffer that `at` elements fit into, so that tensors of other shapes can lie over it."""
    buf = torch.zeros(at, dtype=dtype, device="cuda")
    n = 1
    for s in shape:
        n *= s
    return buf, buf[:n].view(shape)


@pytest.mark.parametrize("dtype", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("batch,ci,co", [(200, 160, 160), (300, 264, 96), (70, 61, 130)])
def test_dense(pcb, dtype, batch, ci, co):
    t, tol = TYPES[dtype]
    xs, ws, ys = (4 * batch, ci), (4, ci, co), (4 * batch, co)
    room = 4 * batch * max(ci, co)
    x, w, dy = _normal(1, xs, t), _normal(2, ws, t, 0.05), _normal(3, ys, t)
    fwd = pcb.DenseFwdDescriptor(xs, ws, pcb.Algebra.QUATERNION, pcb.FilterLayout.IO, False)
    bwd = pcb.DenseBwdDescriptor(xs, ws, pcb.Algebra.QUATERNION, pcb.FilterLayout.IO, True)
    y, dw, dx = torch.empty_like(dy), torch.empty_like(w), torch.empty_like(x)
    pcb.denseFwd(x, w, None, y, fwd)
    pcb.denseBwd(x, w, dy, dw, dx, bwd)
    for _ in range(3):
        buf, x2 = _inside(xs, room, t)                                      # y over x
        x2.copy_(x)
        y2 = buf[:dy.numel()].view(ys)
        pcb.denseFwd(x2, w, None, y2, fwd)
        _close(y2, y, tol)
        x2, dw2 = x.clone(), torch.empty_like(w)                            # dx over x
        pcb.denseBwd(x2, w, dy, dw2, x2, bwd)
        _close(x2, dx, tol)
        _close(dw2, dw, tol)
        buf, dy2 = _inside(ys, room, t)                                     # dx over dy
        dy2.copy_(dy)
        dx2, dw2 = buf[:x.numel()].view(xs), torch.empty_like(w)
        pcb.denseBwd(x, w, dy2, dw2, dx2, bwd)
        _close(dx2, dx, tol)
        _close(dw2, dw, tol)


# few tiles and a long reduction: the fp32 kernel cuts it and adds into a cleared output
@pytest.mark.parametrize("n,c,h,w", [(2, 64, 8, 8), (1, 48, 14, 9), (3, 96, 7, 7)])
def test_fp32_convolution(pcb, n, c, h, w):
    t, tol = TYPES["f32"]
    xs, ws = (4 * n, c, h, w), (4, c, c, 3, 3)
    args = (xs, ws, 1, 1, pcb.Padding.SAME, (), 1, pcb.Algebra.QUATERNION, pcb.DataFormat.NCHW, pcb.FilterLayout.OIHW)
    fwd, bwd = pcb.Conv2DFwdDescriptor(*args, False), pcb.Conv2DBwdDescriptor(*args, True)
    x, f, dy = _normal(1, xs, t), _normal(2, ws, t, 0.04), _normal(3, xs, t)
    y, dw, dx = torch.empty_like(x), torch.empty_like(f), torch.empty_like(x)
    pcb.conv2DFwd(x, f, None, y, fwd)
    pcb.conv2DBwd(x, f, dy, dw, dx, bwd)
    for _ in range(3):
        x2 = x.clone()
        pcb.conv2DFwd(x2, f, None, x2, fwd)
        _close(x2, y, tol)
        for target in ("x", "dy"):
            a, b, dw2 = x.clone(), dy.clone(), torch.empty_like(f)
            pcb.conv2DBwd(a, f, b, dw2, a if target == "x" else b, bwd)
            _close(a if target == "x" else b, dx, tol)
            _close(dw2, dw, tol)


@pytest.mark.parametrize("layout", ["nchw", "nhwc"])
def test_strided_backward(pcb, layout):
    t, tol = TYPES["f16"]
    nhwc = layout == "nhwc"
    n, c, h, w = 6, 32, 40, 36
    xs, ys = ((4 * n, h, w, c), (4 * n, h // 2, w // 2, c)) if nhwc else ((4 * n, c, h, w), (4 * n, c, h // 2, w // 2))
    ws = (4, c, 3, 3, c) if nhwc else (4, c, c, 3, 3)
    bwd = pcb.Conv2DBwdDescriptor(xs, ws, 2, 1, pcb.Padding.SAME, (), 1, pcb.Algebra.QUATERNION, pcb.DataFormat.NHWC if nhwc else pcb.DataFormat.NCHW,
                                  pcb.FilterLayout.OHWI if nhwc else pcb.FilterLayout.OIHW, True)
    x, f, dy = _normal(1, xs, t), _normal(2, ws, t, 0.05), _normal(3, ys, t)
    dw, dx = torch.empty_like(f), torch.empty_like(x)
    pcb.conv2DBwd(x, f, dy, dw, dx, bwd)
    for _ in range(3):
        x2, dw2 = x.clone(), torch.empty_like(f)                            # dx over x
        pcb.conv2DBwd(x2, f, dy, dw2, x2, bwd)
        _close(x2, dx, tol)
        _close(dw2, dw, tol)
        buf = torch.zeros(x.numel(), dtype=t, device="cuda")                # dx over dy
        dy2 = buf[:dy.numel()].view(ys)
        dy2.copy_(dy)
        dx2, dw2 = buf.view(xs), torch.empty_like(f)
        pcb.conv2DBwd(x, f, dy2, dw2, dx2, bwd)
        _close(dx2, dx, tol)
