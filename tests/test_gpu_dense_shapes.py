"""The dense kernels that read the caller's tensors directly, at the sizes where their tiles end: feature counts of every
alignment (1, 2, 4, 8 elements), batches and features around the 128-row, 32- and 64-column tiles and the 64- / 32-element
chunks of the reduced dimension, every cluster split, the wide tile, and the first fp32 sizes beyond their range."""
import numpy as np
import pytest
import torch

from helpers import normal, rel_err, uniform

pytestmark = pytest.mark.gpu

# batch, input features, output features
SHAPES = [
    (1, 1, 1), (1, 8, 8), (5, 7, 9), (31, 66, 127), (33, 64, 130), (128, 128, 250), (65, 129, 33), (257, 100, 68), (40, 1000, 36), (9, 36, 1031),
    (1100, 24, 770),       # more tiles than SMs: the 64-column tile (16-bit)
    (600, 520, 300),
]


@pytest.fixture(scope="module")
def gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import gpu_util
    return gpu_util


def _case(gpu, oracle, shape, dtype, oi):
    b, i, o = shape
    x = gpu.rounded(normal(71, (4 * b, i)), dtype)
    w = gpu.rounded(normal(72, (4, o, i) if oi else (4, i, o), std=(2.0 / (4 * i)) ** 0.5), dtype)
    bias = gpu.rounded(uniform(73, (4, o)), dtype)
    dy = gpu.rounded(normal(74, (4 * b, o)), dtype)
    y = gpu.run_dense_fwd(x, w, bias, oi, dtype, "16p", "tensor")
    dw, dx = gpu.run_dense_bwd(x, w, dy, oi, dtype, "16p", "tensor", True)
    rdw, rdx = oracle.dense_bwd(x, w, dy, oi)
    for got, ref, what in ((y, oracle.dense_fwd(x, w, bias, oi), "y"), (dw, rdw, "dw"), (dx, rdx, "dx")):
        assert np.all(np.isfinite(got)), what
        # fp32: 1e-5; 16-bit results: half a unit in the last place of the stored value (2^-11 / 2^-8 of at most max|ref|),
        # twice for the sums' own error
        tol = {"f32": 1e-5, "f16": 2.0 ** -10, "bf16": 2.0 ** -7}[dtype]
        assert rel_err(got, ref) <= tol, (what, rel_err(got, ref))
    dw2, none = gpu.run_dense_bwd(x, w, dy, oi, dtype, "16p", "tensor", False)   # without the input gradient: the same dw
    assert none is None and rel_err(dw2, dw) <= (1e-5 if dtype == "f32" else 2.0 ** -7)


@pytest.mark.parametrize("dtype", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("oi", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_dense_tile_edges(gpu, oracle, shape, dtype, oi):
    _case(gpu, oracle, shape, dtype, oi)


@pytest.mark.parametrize("shape", [(3, 2048, 24), (3, 2056, 24), (2056, 8, 12)])
def test_dense_fp32_longest_reductions(gpu, oracle, shape):
    _case(gpu, oracle, shape, "f32", False)
