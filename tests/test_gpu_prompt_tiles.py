"""Prompt-sized products at the edges of the column tiles (16 columns, two accumulators up to 128, 256, two halves of 192), with row
tiles that the last one of a matrix does not fill, alone and as a group over the same activations."""
import numpy as np
import pytest

from helpers import Model, close
from oracle.bindings import Q4_K, Q8_0
from tensorlisp_b200 import graph as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ty", [Q4_K, Q8_0])
@pytest.mark.parametrize("K,M,N", [(256, [100], 65), (512, [130, 40, 257], 97), (768, [128 * 60, 128 * 60], 333), (512, [9000, 9500], 385), (256, [128 * 149], 129),
                                   (1280, [300, 129], 257), (512, [128 * 40], 1100)])
def test_tiles(oracle, ty, K, M, N):
    rng = np.random.default_rng(K + sum(M) + N)
    X = rng.standard_normal((N, K)).astype(np.float32)
    ws = [oracle.quantize(ty, (rng.standard_normal((m, K)) * 0.02).astype(np.float32)) for m in M]
    g = G.Graph()
    x = g.input(G.F32, [K, N], "x")
    for j, m in enumerate(M):
        g.output(g.mul_mat(g.weight(ty, [K, m], "w%d" % j), x, "y%d" % j))
    m = Model(g, ws)
    got = m.run(X)
    for y, w, rows in zip(got, ws, M):
        close(y.reshape(N, rows), oracle.mul_mat(ty, w, K, X), 1e-3)
    m.close()


# Few row tiles: their K is cut (into stretches of unequal length where it does not divide), a ragged last row tile and column tile among the parts.
@pytest.mark.parametrize("ty", [Q4_K, Q8_0])
@pytest.mark.parametrize("K,M,N", [(1792, [100], 65), (2816, [300, 40], 130), (5120, [257], 333), (4096, [513, 256, 31], 200), (3328, [1000], 390), (14336, [4000], 70)])
def test_cut_tiles(oracle, ty, K, M, N):
    test_tiles(oracle, ty, K, M, N)
