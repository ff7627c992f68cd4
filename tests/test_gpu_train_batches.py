"""The tensor-core training kernels at batches of one tile, an odd number of tiles and an odd split of the weight gradients."""
import numpy as np
import pytest

from oracle import mlp_oracle as MO
from outbreaklab_b200 import surrogate as S
from test_gpu_mlp import _norm_for, _synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [128, 384, 1152, 2176])
def test_gradient_at_edge_batches(native, n):
    """1, 3, 9 and 17 tiles of 128 samples; the weight gradients split the batch 2, 6, 9 and 2 ways. Against the float64
    restatement that rounds to bf16 at the same points: a sample's operand may round the other way, which moves its term by
    at most 2^-8, and so no block's norm by more than that fraction."""
    net = S.MicroSurrogate(seed=3)
    pairs = _synthetic(100 + n, n)
    norm = _norm_for(pairs)
    net.set_norm(norm)
    params = (np.random.default_rng(n).standard_normal(S.NPARAM) * 0.1).astype(np.float32)
    net.set_params(params)
    loss, g = net.grad(pairs)
    lb, gb = MO.loss_and_grad_bf16(params.astype(np.float64), pairs.astype(np.float64), norm.astype(np.float64))
    assert abs(loss - lb) <= 2.0 ** -8 * abs(lb), (loss, lb)
    o = 0
    for name, shp in MO.SHAPES:
        m = int(np.prod(shp))
        a, b = g[o:o + m].astype(np.float64), gb[o:o + m]
        assert np.linalg.norm(a - b) <= 2.0 ** -8 * np.linalg.norm(b) + 1e-12, (name, np.linalg.norm(a - b) / np.linalg.norm(b))
        o += m
