"""Dense layers whose tiles ask for about as many clusters of 8 CTAs as a device holds at once (15 to 17 on one of 148 SMs): the split of the reduced
dimension falls on either side of that number, and with an SM margin on the other one."""
import numpy as np
import pytest
import torch

from helpers import normal, rel_err

pytestmark = pytest.mark.gpu

# half a unit in the last place of a 16-bit result, twice for the sums' own error; fp32 as elsewhere
TOL = {"f32": 1e-5, "f16": 2.0 ** -10, "bf16": 2.0 ** -7}


@pytest.mark.parametrize("margin", [0, 3])
@pytest.mark.parametrize("dtype,batch,i,o", [("f16", 42, 144, 946), ("bf16", 246, 224, 212), ("f32", 255, 72, 150), ("f16", 32, 144, 1930), ("f16", 64, 40, 1000), ("f32", 42, 144, 946)])
def test_around_a_round_of_clusters(oracle, dtype, batch, i, o, margin):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import gpu_util as gpu
    from phoenix_core_b200 import ops
    x, w = gpu.rounded(normal(81, (4 * batch, i)), dtype), gpu.rounded(normal(82, (4, i, o), std=(2.0 / (4 * i)) ** 0.5), dtype)
    b, dy = gpu.rounded(normal(83, (4, o), std=0.1), dtype), gpu.rounded(normal(84, (4 * batch, o)), dtype)
    ops.setSmMargin(margin)
    try:
        y = gpu.run_dense_fwd(x, w, b, False, dtype, "16p", "tensor")
        dw, dx = gpu.run_dense_bwd(x, w, dy, False, dtype, "16p", "tensor")
    finally:
        ops.setSmMargin(0)
    rdw, rdx = oracle.dense_bwd(x, w, dy)
    for got, want, what in ((y, oracle.dense_fwd(x, w, b), "y"), (dw, rdw, "dw"), (dx, rdx, "dx")):
        assert np.all(np.isfinite(got)) and rel_err(got, want) <= TOL[dtype], (what, rel_err(got, want))
