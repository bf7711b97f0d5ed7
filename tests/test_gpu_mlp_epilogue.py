"""The GEMM epilogue's 16-byte path over the widths where it can go wrong (one
group of 16 columns past a 256-wide tile, a padded row, rows about the 128-row
tile), and gradients that reach the caller directly (a width that is a multiple
of 32) or through the unpadding copy, twice with the same network.  Tolerances
of the other network tests: the oracle rounds the same operands to BF16."""
import numpy as np
import pytest

from oracle import mlp as OM
from shell_gb300 import lib as L
from tests.test_mlp import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,n", [([32, 32, 16], 1), ([8, 288, 257, 40], 127), ([33, 272, 256, 520], 129),
                                    ([8, 64, 7686], 256)])
def test_gradients(cuda_ok, dims, n):
    rng = np.random.default_rng(n)
    net = L.MLP(dims, max_batch=256, seed=3)
    params = [(W, 0.05 * rng.standard_normal(b.shape)) for W, b in net.get_params()]
    net.set_params(params)
    params = [(W.astype(np.float32).astype(np.float64), b.astype(np.float32).astype(np.float64)) for W, b in params]
    for _ in range(2):
        X = rng.standard_normal((n, dims[0])).astype(np.float32)
        T = rng.standard_normal((n, dims[-1])).astype(np.float32)
        loss, dW, db = net.gradients(X, T)
        lo, dWo, dbo = OM.loss_and_gradients(params, X, T, bf16_ops=True)
        assert abs(loss - lo) <= 1e-5 * lo
        for l in range(len(dims) - 1):
            assert rel(dW[l], dWo[l]) < 5e-3, l
            assert rel(db[l], dbo[l]) < 5e-3, l
    net.close()
