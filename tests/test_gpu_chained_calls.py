"""Calls that follow one another on a stream without a pause, each reading what the one in front of it has just written into buffers that
are used again and again: the kernels of a call may be resident while the last kernel of the call in front still writes. The same
calls separated by a synchronisation give the same results (up to the order of the fp32 sums where a kernel adds atomically)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

TYPES = {"f32": (torch.float32, 1e-5), "f16": (torch.float16, 2.0 ** -9), "bf16": (torch.bfloat16, 2.0 ** -6)}


@pytest.fixture(scope="module")
def pcb():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import phoenix_core_b200
    return phoenix_core_b200


def _normal(seed, shape, dtype, std):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(shape, generator=gen, device="cuda") * std).to(dtype)


class _Chain:
    """A 3x3 layer of c channels, a second one on its output, a dense layer on the pooled (here: first) pixels, and their gradients, all
    in the same buffers for every round."""

    def __init__(self, pcb, dtype, c, hw, n):
        self.pcb, self.n, self.c = pcb, n, c
        t = TYPES[dtype][0]
        q, P = pcb.Algebra.QUATERNION, pcb.Padding.SAME
        xs, ws = (4 * n, c, hw, hw), (4, c, c, 3, 3)
        args = (xs, ws, 1, 1, P, (), 1, q, pcb.DataFormat.NCHW, pcb.FilterLayout.OIHW)
        self.fwd, self.bwd = pcb.Conv2DFwdDescriptor(*args, False), pcb.Conv2DBwdDescriptor(*args, True)
        features = hw * hw
        ds, dw = (4 * n * c, features), (4, features, features)            # every channel plane is a batch row
        self.dfwd = pcb.DenseFwdDescriptor(ds, dw, q, pcb.FilterLayout.IO, False)
        self.dbwd = pcb.DenseBwdDescriptor(ds, dw, q, pcb.FilterLayout.IO, True)
        std = (1.0 / (4 * c * 9)) ** 0.5
        self.w1, self.w2 = _normal(1, ws, t, std), _normal(2, ws, t, std)
        self.wd = _normal(3, dw, t, (1.0 / (4 * features)) ** 0.5)
        self.x = torch.empty(xs, dtype=t, device="cuda")
        self.a, self.b, self.g, self.h = (torch.empty_like(self.x) for _ in range(4))
        self.z, self.dz = (torch.empty(ds, dtype=t, device="cuda") for _ in range(2))
        self.dw1, self.dw2, self.dwd = torch.empty_like(self.w1), torch.empty_like(self.w2), torch.empty_like(self.wd)
        self.inputs = [_normal(10 + i, xs, t, 1.0) for i in range(4)]

    def round(self, i, pause):
        p, ds = self.pcb, self.z.shape
        steps = [lambda: self.x.copy_(self.inputs[i % 4]),
                 lambda: p.conv2DFwd(self.x, self.w1, None, self.a, self.fwd),
                 lambda: p.conv2DFwd(self.a, self.w2, None, self.b, self.fwd),
                 lambda: p.denseFwd(self.b.view(ds), self.wd, None, self.z, self.dfwd),
                 lambda: p.denseBwd(self.b.view(ds), self.wd, self.z, self.dwd, self.dz, self.dbwd),
                 lambda: p.conv2DBwd(self.a, self.w2, self.dz.view(self.x.shape), self.dw2, self.g, self.bwd),
                 lambda: p.conv2DBwd(self.x, self.w1, self.g, self.dw1, self.h, self.bwd)]
        for step in steps:
            step()
            if pause:
                torch.cuda.synchronize()
        return [t.clone() for t in (self.a, self.b, self.z, self.dz, self.g, self.h, self.dwd, self.dw2, self.dw1)]


@pytest.mark.parametrize("stream", ["default", "side"])
@pytest.mark.parametrize("dtype,c,hw,n", [("f16", 16, 16, 4), ("f16", 40, 9, 3), ("bf16", 64, 14, 8), ("f32", 16, 12, 4), ("f32", 64, 7, 2)])
def test_chained_calls(pcb, dtype, c, hw, n, stream):
    tol = TYPES[dtype][1]
    side = torch.cuda.Stream() if stream == "side" else torch.cuda.current_stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        chain = _Chain(pcb, dtype, c, hw, n)
        want = [chain.round(i, True) for i in range(4)]
        got = [chain.round(i, False) for i in range(24)]
        torch.cuda.synchronize()
    for i, tensors in enumerate(got):
        for k, (a, b) in enumerate(zip(tensors, want[i % 4])):
            a, b = a.double(), b.double()
            assert torch.isfinite(a).all()
            assert ((a - b).abs().max() / b.abs().max()).item() <= tol, (i, k)
