"""Plain rows straight into the operand of the prompt products: lengths that end inside a strip of four blocks, row counts that end
inside a group of eight, enough of both to take the eight-column kernel."""
import numpy as np
import pytest

from helpers import Model, close
from oracle.bindings import Q4_K, Q8_0
from tensorlisp_b200 import graph as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ty", [Q4_K, Q8_0])
@pytest.mark.parametrize("K,N", [(256, 2400), (1280, 1187), (4096, 601), (9216, 260)])
def test_rows(oracle, ty, K, N):
    rng = np.random.default_rng(K + N)
    X = (rng.standard_normal((N, K)) * np.exp(rng.standard_normal((N, 1)))).astype(np.float32)
    X[N // 2] = 0
    X[1, : K // 2] = 0
    W = (rng.standard_normal((40, K)) * 0.02).astype(np.float32)
    Wq = oracle.quantize(ty, W)
    g = G.Graph()
    x = g.input(G.F32, [K, N], "x")
    w = g.weight(ty, [K, 40], "w")
    g.output(g.mul_mat(w, x, "all"))
    m = Model(g, [Wq])
    (got,) = m.run(X)
    want = oracle.mul_mat(ty, Wq, K, X)
    for n in range(0, N, 37):   # column by column: their sizes differ
        close(got.reshape(N, 40)[n], want[n], 1.5e-3)
    close(got.reshape(N, 40)[N - 1], want[N - 1], 1.5e-3)
    assert not got.reshape(N, 40)[N // 2].any()
    m.close()
