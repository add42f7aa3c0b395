"""f16 / bf16 weight matrices on the tensor cores: the activations keep their f32 precision (three terms of the weights'
type), so the result agrees with the f64 product like an f32 sum does. Sizes at the edges of tiles (128 rows), boxes (64
weights), steps (128), chunks (128 or 256), column groups (8 .. 80 per pass) and CTA stretches."""
import numpy as np
import pytest

from helpers import Model
from tensorlisp_b200 import graph as G

pytestmark = pytest.mark.gpu


def _bf16(w):
    u = w.view(np.uint32)
    r = ((u + 0x7fff + ((u >> 16) & 1)) >> 16).astype(np.uint16)
    return r, (r.astype(np.uint32) << 16).view(np.float32)


@pytest.mark.parametrize("ty", [G.F16, G.BF16])
@pytest.mark.parametrize("K,M,N", [(64, 1, 1), (64, 128, 8), (72, 129, 9), (200, 300, 3), (256, 127, 16), (1000, 777, 17), (1024, 500, 24), (1160, 385, 25),
                                   (4096, 1000, 48), (512, 2500, 49), (4104, 260, 80), (640, 20000, 1), (640, 1100, 81), (2048, 19000, 5), (448, 384, 300)])
def test_against_f64(ty, K, M, N):
    rng = np.random.default_rng(K + M + N)
    W = (rng.standard_normal((M, K)) * 0.02).astype(np.float32)
    # columns of very different size, with a wide spread inside each
    X = (rng.standard_normal((N, K)) * np.exp(rng.standard_normal((N, K)) * 2) * np.exp(rng.standard_normal((N, 1)) * 8)).astype(np.float32)
    X[0, : min(K, 5)] = 0
    if ty == G.F16:
        stored = W.astype(np.float16)
        value = stored.astype(np.float64)
    else:
        stored, value = _bf16(W)
        value = value.astype(np.float64)
    g = G.Graph()
    y = g.output(g.mul_mat(g.weight(ty, [K, M], "W"), g.input(G.F32, [K, N], "x"), "y"))
    m = Model(g, [stored])
    for _ in range(2):
        (got,) = m.run(X)
    want = X.astype(np.float64) @ value.T
    # a sum of K products rounded to f32: 1e-6 of the sum of their magnitudes at most
    bound = 1e-6 * (np.abs(X.astype(np.float64)) @ np.abs(value).T) + 1e-37
    assert (np.abs(got.reshape(N, M) - want) <= bound).all()
    m.close()


def test_values_that_are_not_finite_stay_in_their_column():
    K, M, N = 512, 130, 3
    rng = np.random.default_rng(1)
    W = (rng.standard_normal((M, K)) * 0.02).astype(np.float16)
    X = rng.standard_normal((N, K)).astype(np.float32)
    X[1, 7] = np.inf
    g = G.Graph()
    g.output(g.mul_mat(g.weight(G.F16, [K, M], "W"), g.input(G.F32, [K, N], "x"), "y"))
    m = Model(g, [W])
    (got,) = m.run(X)
    got = got.reshape(N, M)
    for n in (0, 2):
        assert np.abs(got[n] - X[n].astype(np.float64) @ W.astype(np.float64).T).max() < 1e-4
    assert not np.isfinite(got[1]).any()
    m.close()
