"""Network kernels on numbers that every step represents exactly.

Small integers: products and sums are exact in FP32, activations of 8 and more
pass the GELU unchanged with slope 1, and every BF16 operand is an integer of at
most 256 (gradients: times a power of two, rows times outputs being one).  The
results then equal the integer arithmetic, bit for bit: a column, row or bias that
an epilogue, a transpose, a partial sum or a copy drops or misplaces shows, where
a relative bound over the whole matrix would not see it."""
import numpy as np
import pytest

from shell_gb300 import lib as L

pytestmark = pytest.mark.gpu


def _network(dims, rng):
    """Weights and inputs whose activations stay between 8 and 256."""
    params = []
    for l in range(len(dims) - 1):
        W = np.zeros((dims[l + 1], dims[l]), dtype=np.float32)
        for r in range(dims[l + 1]):
            W[r, rng.integers(0, dims[l], 2)] = 1.0
        if l == len(dims) - 2:
            W *= rng.choice([-1.0, 1.0], W.shape).astype(np.float32)
        params.append((W, rng.integers(8, 12, dims[l + 1]).astype(np.float32)))
    return params


def _forward(params, X):
    H = [X.astype(np.float64)]
    for l, (W, b) in enumerate(params):
        H.append(H[-1] @ W.astype(np.float64).T + b)
        if l < len(params) - 1:
            assert H[-1].min() >= 8 and H[-1].max() <= 256
    return H


@pytest.mark.parametrize("dims,n", [([8, 16, 16], 1), ([33, 257, 272], 127), ([8, 288, 257, 40], 129),
                                    ([9, 64, 256, 7686], 256), ([5, 31], 3)])
def test_predictions(cuda_ok, dims, n):
    rng = np.random.default_rng(n)
    net = L.MLP(dims, max_batch=256, seed=1)
    params = _network(dims, rng)
    net.set_params(params)
    X = rng.integers(0, 4, (n, dims[0])).astype(np.float32)
    assert np.array_equal(net.predict(X).astype(np.float64), _forward(params, X)[-1])
    net.close()


@pytest.mark.parametrize("dims,n", [([8, 16, 16], 1), ([33, 257, 512], 128), ([8, 288, 257, 32], 64),
                                    ([9, 64, 256, 1024], 256)])
def test_gradients(cuda_ok, dims, n):
    rng = np.random.default_rng(n)
    net = L.MLP(dims, max_batch=256, seed=1)
    params = _network(dims, rng)
    net.set_params(params)
    X = rng.integers(0, 4, (n, dims[0])).astype(np.float32)
    H = _forward(params, X)
    D = rng.integers(-2, 3, H[-1].shape).astype(np.float64)
    loss, dW, db = net.gradients(X, (H[-1] - D).astype(np.float32))
    assert loss == np.mean(D * D)
    G = D * 2.0 / D.size
    for l in reversed(range(len(params))):
        assert np.array_equal(dW[l].astype(np.float64), G.T @ H[l]), l
        assert np.array_equal(db[l].astype(np.float64), G.sum(axis=0)), l
        G = G @ params[l][0].astype(np.float64)
        assert np.abs(G).max() * D.size / 2.0 <= 256
    net.close()


@pytest.mark.parametrize("M,N,K", [(130, 257, 72), (128, 256, 64), (129, 519, 640), (77, 201, 136)])
def test_product(cuda_ok, M, N, K):
    rng = np.random.default_rng(M)
    A, B = (rng.integers(-8, 9, s).astype(np.float32) for s in ((M, K), (N, K)))
    bits = [np.ascontiguousarray(x.view(np.uint32) >> 16).astype(np.uint16) for x in (A, B)]  # exact in BF16
    C = L.gemm_bf16(*bits)
    assert np.array_equal(C.astype(np.float64).reshape(M, N), A.astype(np.float64) @ B.astype(np.float64).T)
