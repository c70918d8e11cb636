"""GPU: the training kernels (mlp_train.cu) against the CPU oracle at the edges of their blocks:
one row, a ragged block of 32 rows, a ragged last split of the weight gradients.

FP32 sums of at most 4,097 products behind four layers: about sqrt(4097) 2^-24 = 4e-6 of a
gradient's norm a layer; held to 1e-4, as the other comparison of these kernels."""
import numpy as np
import pytest

import mlp_oracle as mo
from sps_gb300 import surrogate as sg
from test_gpu_surrogate import layer_errors, random_tuples

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 31, 33, 257, 4097])
def test_gradients_at_block_edges(built_gpu, rows):
    net = sg.Mlp(batch=4160, seed=5, quantize=False)
    p = net.params().astype(np.float64)
    t = random_tuples(np.random.default_rng(rows), rows)
    loss, g = net.grad(t)
    loss_ref, g_ref = mo.loss_grad(p, t.astype(np.float64), quantize=False)
    assert abs(loss - loss_ref) <= 1e-4 * loss_ref
    assert max(layer_errors(g, g_ref)) <= 1e-4
    net.close()
