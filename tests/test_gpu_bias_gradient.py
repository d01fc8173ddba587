"""Bias gradients (column sums over the batch, 32 rows at a time) for batches of
one, a few and many rows a warp, and output widths of different blocks.

Reference: the network's oracle.  Tolerance: relative L2 <= 5e-3, as for all
gradients of a batch (BF16 activations and output gradients)."""
import numpy as np
import pytest

from tests.conftest import rel_l2
from tests.test_gpu_surrogate import _random_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kz,batch", [(5, 128), (13, 256), (20, 1152)])
def test_bias_gradients(gpu_lib, kz, batch):
    from oracle import mlp_oracle as mo
    sur = gpu_lib.Surrogate(kz, capacity=2 * batch, batch=batch, seed=3)
    d = sur.dims()
    rng = np.random.default_rng(5)
    P = _random_params(sur, rng, scale=1.5)
    X = np.zeros((batch, d["kin"]), np.float32)
    X[:, :d["nin"]] = rng.normal(size=(batch, d["nin"]))
    T = np.zeros((batch, d["nop"]), np.float32)
    T[:, :d["nout"]] = rng.normal(size=(batch, d["nout"]))
    _, grads = mo.backward(P, X, T, d["nout"])
    for layer in (0, 3):
        _, _, gb = sur.gradients(X, T, layer)
        assert rel_l2(gb, grads[layer][1]) <= 5e-3, layer
    sur.close()
