"""Cases for timing the quaternion operators through the entry points a program calls: conv2DFwd / conv2DBwd,
denseFwd / denseBwd and one training step of the quaternion ResNet-18.

A case is a dict of plain values; `prepare` builds the tensors and descriptors that a program keeps, `run` makes one pass.
Activations and output gradients are N(0, 1), filters He-normal over their real inputs, as in the benchmark.

  op      "conv", "dense" or "resnet"
  mode    "fwd" (inference: the forward call alone) or "train" (forward, filter gradient and, unless the input is
          real-valued, input gradient)
  dtype   "f32", "f16" or "bf16"
"""
import math

import torch
import torch.nn.functional as F

import phoenix_core_b200 as pcb
from phoenix_core_b200.qresnet import LOSS_SCALE, QResNet18

DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
LEARNING_RATE = 0.1                  # the harness's


def _conv(name, dtype, mode, n, ci, co, h, w, k, stride=1, layout="nchw", bias=False, real=False):
    return {"name": name, "op": "conv", "mode": mode, "dtype": dtype, "n": n, "ci": ci, "co": co, "h": h, "w": w, "k": k,
            "stride": stride, "layout": layout, "bias": bias, "real": real}


def _dense(name, dtype, mode, n, ci, co, bias=True):
    return {"name": name, "op": "dense", "mode": mode, "dtype": dtype, "n": n, "ci": ci, "co": co, "bias": bias}


def listed():
    return [
        # a single small layer evaluated in full precision: latency and launches
        _conv("conv3x3_16at32_f32_fwd", "f32", "fwd", 8, 16, 16, 32, 32, 3),
        # the classifier of the quaternion ResNet-18 (1000 classes = 250 quaternion outputs) in training
        _dense("dense_128to250_f16_train", "f16", "train", 128, 128, 250),
        # a wide dense layer trained in full precision
        _dense("dense_512to512_f32_train", "f32", "train", 256, 512, 512),
        # inference on images that are neither square nor a round number of pixels, with a bias
        _conv("conv3x3_24to40at45x37_f16_fwd", "f16", "fwd", 10, 24, 40, 45, 37, 3, bias=True),
        # the benchmark's layer: a wide pointwise convolution on large planes
        _conv("conv1x1_128to256at56_f16_train", "f16", "train", 64, 128, 256, 56, 56, 1),
        # a deep pointwise layer: 14 x 14 planes, whose rows and planes are not a round number of bytes
        _conv("conv1x1_256at14_bf16_train", "bf16", "train", 128, 256, 256, 14, 14, 1),
        # the 3x3 layer of an early residual stage, channels-first and channels-last
        _conv("conv3x3_64at56_f16_train", "f16", "train", 128, 64, 64, 56, 56, 3),
        _conv("conv3x3_64at56_nhwc_f16_train", "f16", "train", 128, 64, 64, 56, 56, 3, layout="nhwc"),
        # the down-sampling 3x3 layer of a middle stage
        _conv("conv3x3s2_128at28_f16_train", "f16", "train", 128, 128, 128, 28, 28, 3, stride=2),
        # a middle stage's 3x3 layer in full precision, the default policy of the engine
        _conv("conv3x3_128at28_f32_train", "f32", "train", 128, 128, 128, 28, 28, 3),
        # the network's stem: RGB images as real-valued quaternions, 7x7 stride 2, no input gradient
        _conv("conv7x7s2_3to16at224_f16_train", "f16", "train", 128, 3, 16, 224, 224, 7, stride=2, real=True),
        # a whole training step of the quaternion ResNet-18, replayed as the harness does on one GPU
        {"name": "qresnet18_step_b128", "op": "resnet", "mode": "train", "dtype": "f16", "n": 128, "h": 224},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    """One more case of the listed ranges: channel counts are mostly multiples of 8, planes and batches anything."""
    kind = rng.choice(("conv", "conv", "conv", "conv", "pointwise", "pointwise", "dense", "dense", "stem", "resnet"))
    dtype = rng.choice(("f16", "f16", "bf16", "f32"))
    mode = rng.choice(("train", "train", "fwd"))
    if kind == "resnet":
        case = {"op": "resnet", "mode": "train", "dtype": "f16", "n": rng.randrange(16, 121, 8), "h": rng.choice((96, 128, 160, 192, 224))}
    elif kind == "dense":
        case = _dense(None, dtype, mode, _log_int(rng, 32, 1024), 8 * _log_int(rng, 8, 96), _log_int(rng, 64, 1024), rng.random() < 0.5)
    elif kind == "stem":
        size = 8 * rng.randrange(8, 28)
        case = _conv(None, "f16", "train", _log_int(rng, 8, 127), 3, 8 * rng.randrange(1, 5), size, size, rng.choice((3, 5, 7)), 2, real=True)
    else:
        side = _log_int(rng, 7, 112)
        # wide layers have small planes, as in a residual network: about 64 channels at 56 x 56
        wide = min(512, max(16, 3584 // side))
        ci, co = (8 * _log_int(rng, 2, max(3, wide // 8)) for _ in range(2))
        if rng.random() < 0.15:
            co += rng.randrange(1, 8)
        w = side if rng.random() < 0.6 else max(7, side + rng.randrange(-side // 4, side // 4 + 1))
        nhwc = dtype != "f32" and kind == "conv" and rng.random() < 0.25
        case = _conv(None, dtype, mode, _log_int(rng, 4, 128), ci, co, side, w, 1 if kind == "pointwise" else rng.choice((3, 3, 3, 5)),
                     rng.choice((1, 1, 1, 2)), "nhwc" if nhwc else "nchw", rng.random() < 0.3)
    case.pop("name", None)
    # no costlier than the largest listed case of the type
    most = 3e11 if dtype == "f32" else 1.2e12
    while case["op"] == "conv" and work(case)["flops"] > most and case["n"] > 1:
        case["n"] = max(1, case["n"] // 2)
    return case


# ---- geometry -----------------------------------------------------------------------------------------------------------

def _same(size, k, stride):
    """(output size, padding before, padding after) of the SAME rule."""
    out = -(-size // stride)
    total = max((out - 1) * stride + k - size, 0)
    return out, total // 2, total - total // 2


def _conv_args(c):
    planes = (1 if c["real"] else 4) * c["n"]
    nhwc = c["layout"] == "nhwc"
    xshape = (planes, c["h"], c["w"], c["ci"]) if nhwc else (planes, c["ci"], c["h"], c["w"])
    wshape = (4, c["co"], c["k"], c["k"], c["ci"]) if nhwc else (4, c["co"], c["ci"], c["k"], c["k"])
    args = (xshape, wshape, c["stride"], 1, pcb.Padding.SAME, (), 1, pcb.Algebra.QUATERNION,
            pcb.DataFormat.NHWC if nhwc else pcb.DataFormat.NCHW, pcb.FilterLayout.OHWI if nhwc else pcb.FilterLayout.OIHW)
    return xshape, wshape, args


# ---- one pass -----------------------------------------------------------------------------------------------------------

def _normal(gen, shape, std, dtype):
    return (torch.randn(shape, generator=gen, device="cuda") * std).to(dtype)


def _inputs(c, seed):
    """The tensors of a layer case from the seed: x, filters, bias (or None), output gradient (training only)."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype = DTYPES[c["dtype"]]
    if c["op"] == "dense":
        xshape, wshape, yshape, fan = (4 * c["n"], c["ci"]), (4, c["ci"], c["co"]), (4 * c["n"], c["co"]), 4 * c["ci"]
    else:
        xshape, wshape, args = _conv_args(c)
        fan = 4 * c["ci"] * c["k"] ** 2
        yshape = pcb.Conv2DFwdDescriptor(*args, c["bias"], c["real"]).getOutputShape()
    x = _normal(gen, xshape, 1.0, dtype)
    w = _normal(gen, wshape, math.sqrt(2.0 / fan), dtype)
    bias = _normal(gen, (4, c["co"]), 0.1, dtype) if c["bias"] else None
    dy = _normal(gen, yshape, 1.0, dtype) if c["mode"] == "train" else None
    return x, w, bias, dy


def _batch(c, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    images = torch.randn((c["n"], 3, c["h"], c["h"]), generator=gen, device="cuda").to(torch.float16)
    return images, torch.randint(0, 1000, (c["n"],), generator=gen, device="cuda")


def prepare(case, seed):
    c = case
    if c["op"] == "resnet":
        torch.backends.cudnn.enabled = False              # as the harness: nothing falls into another library's convolutions
        images, labels = _batch(c, seed)
        model = QResNet18(torch.device("cuda", torch.cuda.current_device()), seed=seed)
        for _ in range(2):                                # eager steps grow the workspaces; a zero rate leaves the weights
            model.train_step(images, labels, lr=0.0)
        model.flat_mom.zero_()
        model.bn_m.zero_()
        model.capture(images, labels, lr=LEARNING_RATE)
        return {"case": c, "model": model, "images": images, "labels": labels}
    x, w, bias, dy = _inputs(c, seed)
    s = {"case": c, "x": x, "w": w, "bias": bias, "dy": dy}
    train = c["mode"] == "train"
    if c["op"] == "dense":
        args = (tuple(x.shape), tuple(w.shape), pcb.Algebra.QUATERNION, pcb.FilterLayout.IO)
        s["fwd"] = pcb.DenseFwdDescriptor(*args, c["bias"])
        s["bwd"] = pcb.DenseBwdDescriptor(*args, True) if train else None
    else:
        args = _conv_args(c)[2]
        s["fwd"] = pcb.Conv2DFwdDescriptor(*args, c["bias"], c["real"])
        s["bwd"] = pcb.Conv2DBwdDescriptor(*args, not c["real"], c["real"]) if train else None
    s["y"] = torch.empty(s["fwd"].getOutputShape(), dtype=x.dtype, device="cuda")
    s["dw"] = torch.empty_like(w) if train else None
    s["dx"] = torch.empty_like(x) if train and not c.get("real") else None
    return s


def run(state):
    s = state
    c = s["case"]
    if c["op"] == "resnet":
        m = s["model"]
        loss = m.step(s["images"], s["labels"], lr=LEARNING_RATE)
        return {"loss": loss, "weights": m.flat_w32, "bn_weights": m.bn_w}
    forward, backward = (pcb.denseFwd, pcb.denseBwd) if c["op"] == "dense" else (pcb.conv2DFwd, pcb.conv2DBwd)
    forward(s["x"], s["w"], s["bias"], s["y"], s["fwd"])
    if c["mode"] == "fwd":
        return {"y": s["y"]}
    backward(s["x"], s["w"], s["dy"], s["dw"], s["dx"], s["bwd"])
    return {"y": s["y"], "dw": s["dw"], "dx": s["dx"]}


# ---- what a pass cannot do without ----------------------------------------------------------------------------------------

# the convolutions of the network: input and output channels, input size at 224, kernel, stride, how many
NETWORK = ((16, 16, 56, 3, 1, 4), (16, 32, 56, 3, 2, 1), (32, 32, 28, 3, 1, 3), (32, 64, 28, 3, 2, 1), (64, 64, 14, 3, 1, 3),
           (64, 128, 14, 3, 2, 1), (128, 128, 7, 3, 1, 3), (16, 32, 56, 1, 2, 1), (32, 64, 28, 1, 2, 1), (64, 128, 14, 1, 2, 1))


def work(case):
    c = case
    if c["op"] == "resnet":
        n, h = c["n"], c["h"]
        flops, params = 2 * 8.0 * n * (h // 2) ** 2 * 16 * 3 * 49, 4 * (16 * 3 * 49 + 128 * 250 + 250)
        flops += 3 * 32.0 * n * 128 * 250
        for ci, co, size, k, stride, count in NETWORK:
            out = -(-(size * h // 224) // stride)
            flops += count * 3 * 32.0 * n * out * out * co * ci * k * k
            params += count * 4 * co * ci * k * k
        # images, and per parameter: master and momentum read and written, gradient written
        return {"bytes": 2.0 * n * 3 * h * h + 18.0 * params, "flops": flops}
    eb = 4 if c["dtype"] == "f32" else 2
    if c["op"] == "dense":
        ho = wo = h = w = k = 1
    else:
        h, w, k = c["h"], c["w"], c["k"]
        ho, wo = _same(h, k, c["stride"])[0], _same(w, k, c["stride"])[0]
    real = bool(c.get("real"))
    x = (1 if real else 4) * c["n"] * c["ci"] * h * w
    y = 4 * c["n"] * c["co"] * ho * wo
    f = 4 * c["co"] * c["ci"] * k * k
    flops = (8.0 if real else 32.0) * c["n"] * ho * wo * c["co"] * c["ci"] * k * k
    total = x + f + y
    if c["mode"] == "train":                              # dy in, dw out, dx out (x and the filters are read once in all)
        total += y + f + (0 if real else x)
        flops *= 2 if real else 3
    return {"bytes": float(eb * total), "flops": flops}


def tolerance(case):
    """About four times what separates two correct orders of summation: the rounding of the stored results for the
    16-bit types, the accumulation for 32 bits. The training step rounds every activation to 16 bits on its way and sums the
    batch-norm statistics in any order: its gradients differ by 3 to 4 % from run to run (as much as from 64 bits), which
    moves the updated weights by 4e-4 after one step."""
    if case["op"] == "resnet":
        return {"rel": 4e-3}
    return {"rel": {"f32": 1e-5, "f16": 1.2e-3, "bf16": 1e-2}[case["dtype"]]}


# ---- the same in 64 bits ------------------------------------------------------------------------------------------------

# y = x (Hamilton product) w: component l of x times component l ^ d of w goes into component d of y, with these negative
NEGATIVE = {(1, 0), (1, 2), (2, 0), (2, 3), (3, 0), (3, 1)}


def _block(w, real=False):
    """[4, Co, Ci, ...] quaternion filters -> the [4 Co, (4) Ci, ...] real ones that act on the stacked components."""
    rows = [torch.cat([-w[l ^ d] if (l, d) in NEGATIVE else w[l ^ d] for l in range(1 if real else 4)], dim=1) for d in range(4)]
    return torch.cat(rows, dim=0)


def _unblock(g, co, ci, real=False):
    """The gradient of the four filters from the gradient of the block matrix."""
    out = torch.zeros((4, co, ci) + tuple(g.shape[2:]), dtype=g.dtype, device=g.device)
    for d in range(4):
        for l in range(1 if real else 4):
            part = g[d * co:(d + 1) * co, l * ci:(l + 1) * ci]
            out[l ^ d] += -part if (l, d) in NEGATIVE else part
    return out


class _Conv64(torch.autograd.Function):
    """A real SAME convolution in 64 bits, one matrix product per tap and slice of the batch."""

    @staticmethod
    def forward(ctx, x, w, stride):
        n, ci, h, wd = x.shape
        co, k = w.shape[0], w.shape[2]
        ho, top, bottom = _same(h, k, stride)
        wo, left, right = _same(wd, k, stride)
        ctx.save_for_backward(x, w)
        ctx.geom = (stride, ho, wo, (left, right, top, bottom))
        y = torch.zeros((n, co, ho, wo), dtype=x.dtype, device=x.device)
        for i in range(0, n, 32):
            xp = F.pad(x[i:i + 32], ctx.geom[3])
            for a in range(k):
                for b in range(k):
                    part = xp[:, :, a:a + (ho - 1) * stride + 1:stride, b:b + (wo - 1) * stride + 1:stride].reshape(-1, ci, ho * wo)
                    y[i:i + 32] += torch.matmul(w[:, :, a, b], part).view(-1, co, ho, wo)
        return y

    @staticmethod
    def backward(ctx, dy):
        x, w = ctx.saved_tensors
        stride, ho, wo, pad = ctx.geom
        n, ci, h, wd = x.shape
        co, k = w.shape[0], w.shape[2]
        dx, dw = torch.zeros_like(x) if ctx.needs_input_grad[0] else None, torch.zeros_like(w)
        for i in range(0, n, 32):
            xp = F.pad(x[i:i + 32], pad)
            dxp = torch.zeros_like(xp)
            g = dy[i:i + 32].reshape(-1, co, ho * wo)
            for a in range(k):
                for b in range(k):
                    at = (slice(None), slice(None), slice(a, a + (ho - 1) * stride + 1, stride), slice(b, b + (wo - 1) * stride + 1, stride))
                    part = xp[at].reshape(-1, ci, ho * wo)
                    dw[:, :, a, b] += torch.matmul(g, part.transpose(1, 2)).sum(0)
                    if dx is not None:
                        dxp[at] += torch.matmul(w[:, :, a, b].t(), g).view(-1, ci, ho, wo)
            if dx is not None:
                dx[i:i + 32] = dxp[:, :, pad[2]:pad[2] + h, pad[0]:pad[0] + wd]
        return dx, dw, None


def _join(x, n):
    """[4N, C, ...] stacked on the batch axis -> [N, 4C, ...]."""
    return x.view(4, n, *x.shape[1:]).transpose(0, 1).reshape(n, 4 * x.shape[1], *x.shape[2:])


def _split(x):
    """[N, 4C, ...] -> [4N, C, ...]."""
    return x.view(x.shape[0], 4, x.shape[1] // 4, *x.shape[2:]).transpose(0, 1).reshape(4 * x.shape[0], x.shape[1] // 4, *x.shape[2:])


def _exact_layer(c, seed):
    x, w, bias, dy = (t if t is None else t.double() for t in _inputs(c, seed))
    n, real = c["n"], bool(c.get("real"))
    nhwc = c.get("layout") == "nhwc"
    if c["op"] == "dense":
        x, w, dy = x[:, :, None, None], w.transpose(1, 2)[..., None, None], None if dy is None else dy[:, :, None, None]
    elif nhwc:
        x, w, dy = x.permute(0, 3, 1, 2).contiguous(), w.permute(0, 1, 4, 2, 3), None if dy is None else dy.permute(0, 3, 1, 2).contiguous()
    co, ci = w.shape[1], w.shape[2]
    train = c["mode"] == "train"
    xr = (x if real else _join(x, n)).requires_grad_(train and not real)
    wr = _block(w, real).requires_grad_(train)
    y = _Conv64.apply(xr, wr, c.get("stride", 1))
    out = {"y": _split(y.detach())}
    if bias is not None:
        out["y"] = (out["y"].view(4, n, co, -1) + bias[:, None, :, None]).view(out["y"].shape)
    if train:
        y.backward(_join(dy, n))
        out["dw"] = _unblock(wr.grad, co, ci, real)
        out["dx"] = None if real else _split(xr.grad)
    if c["op"] == "dense":
        return {k: v.squeeze(-1).squeeze(-1).transpose(1, 2).contiguous() if k == "dw" else v.flatten(1) for k, v in out.items()}
    if nhwc:
        return {k: v.permute(0, 1, 3, 4, 2).contiguous() if k == "dw" else v.permute(0, 2, 3, 1).contiguous() for k, v in out.items()}
    return out


def _exact_resnet(c, seed):
    """The network of phoenix_core_b200.qresnet in 64 bits, on its 16-bit working copy of the initial weights."""
    images, labels = _batch(c, seed)
    model = QResNet18(torch.device("cuda", torch.cuda.current_device()), seed=seed)
    masters, n = model.flat_w32.double(), c["n"]
    flat = masters.half().double()
    bn_flat = model.bn_w.double()
    flat.requires_grad_(True)
    bn_flat.requires_grad_(True)
    at = bn_at = 0

    def take(*shape):
        nonlocal at
        count = math.prod(shape)
        v = flat[at:at + count].view(shape)
        at += (count + 7) // 8 * 8
        return v

    def conv(x, w, stride, real=False):
        return _split(_Conv64.apply(x if real else _join(x, n), _block(w, real), stride))

    def bn(x, gb):
        mean, var = x.mean(dim=(0, 2, 3), keepdim=True), x.var(dim=(0, 2, 3), keepdim=True, unbiased=False)
        ch = x.shape[1]
        return (x - mean) * torch.rsqrt(var + 1e-5) * gb[:ch].view(1, -1, 1, 1) + gb[ch:].view(1, -1, 1, 1)

    def take_bn(ch):
        nonlocal bn_at
        bn_at += 2 * ch
        return bn_flat[bn_at - 2 * ch:bn_at]

    # parameters lie in the order in which the layers are made
    x = conv(images.double(), take(4, 16, 3, 7, 7), 2, real=True)
    x = F.max_pool2d(torch.relu(bn(x, take_bn(16))), 3, 2, 1)
    cin = 16
    for si, cout in enumerate((16, 32, 64, 128)):
        for bi in range(2):
            stride = 2 if si > 0 and bi == 0 else 1
            w1, g1 = take(4, cout, cin, 3, 3), take_bn(cout)
            w2, g2 = take(4, cout, cout, 3, 3), take_bn(cout)
            short = x
            if stride != 1 or cin != cout:
                wd, gd = take(4, cout, cin, 1, 1), take_bn(cout)
                short = bn(conv(x, wd, stride), gd)
            x = torch.relu(bn(conv(torch.relu(bn(conv(x, w1, stride), g1)), w2, 1), g2) + short)
            cin = cout
    x = _join(x.mean(dim=(2, 3)), n)
    wf, bf = take(4, 128, 250), take(4, 250)
    logits = x @ _block(wf.transpose(1, 2)).t() + bf.reshape(-1)
    loss = F.cross_entropy(logits, labels)
    (loss * LOSS_SCALE).backward()
    step = LEARNING_RATE / LOSS_SCALE
    return {"loss": loss.detach(), "weights": masters - step * flat.grad, "bn_weights": bn_flat.detach() - step * bn_flat.grad}


def exact(case, seed):
    return _exact_resnet(case, seed) if case["op"] == "resnet" else _exact_layer(case, seed)
