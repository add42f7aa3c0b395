"""MUL_MAT through compiled programs against the oracle (= the reference's CPU backend semantics:
activations quantized to Q8_0 / Q8_K, integer block dots, f32 scaling).
Bar: max|got-want| <= 1e-3 * max|want| (the bar the benchmark sets); observed ~1e-6 (summation order)."""
import os

import numpy as np
import pytest

from helpers import Model, close
from oracle.bindings import F16, F32, Q4_0, Q4_K, Q8_0
from tensorlisp_b200 import graph as G
from tensorlisp_b200.native import TlbError

pytestmark = pytest.mark.gpu
GOLD = np.load(os.path.join(os.path.dirname(__file__), "golden", "golden.npz"))
TYPES = [(Q8_0, "q8_0"), (Q4_0, "q4_0"), (Q4_K, "q4_K")]
TOL = 1e-3


def mm_model(ty, K, M, N, Wq):
    g = G.Graph()
    w = g.weight(ty, [K, M], "W")
    x = g.input(G.F32, [K, N], "x")
    y = g.output(g.mul_mat(w, x, "y"))
    return Model(g, [Wq]), y


@pytest.mark.parametrize("ty,name", TYPES)
def test_golden(ty, name, oracle):
    Wq = oracle.quantize(ty, GOLD["mm_w"])
    m, _ = mm_model(ty, 512, 24, 5, Wq)
    (y,) = m.run(GOLD["mm_x"])
    close(y, GOLD["mm_y_" + name], TOL)
    m.close()


@pytest.mark.parametrize("ty,name", TYPES)
@pytest.mark.parametrize("K,M", [(4096, 512), (14336, 64), (256, 96), (1024, 7)])
@pytest.mark.parametrize("N", [1, 2, 3, 5, 8, 9, 16, 23, 32, 40, 70, 129])
def test_shapes(oracle, ty, name, K, M, N):
    rng = np.random.default_rng(K + M + N)
    W = (rng.standard_normal((M, K)) * 0.02).astype(np.float32)
    X = rng.standard_normal((N, K)).astype(np.float32)
    Wq = oracle.quantize(ty, W)
    m, _ = mm_model(ty, K, M, N, Wq)
    (y,) = m.run(X)
    err = close(y, oracle.mul_mat(ty, Wq, K, X), TOL)
    if name in ("q8_0", "q4_K") and N > 64:
        # prompt-sized batches: weights and activations as scaled f16 operands (two f16 roundings per product)
        assert err <= 5e-4 * np.abs(y).max() + 1e-6
    else:
        assert err <= 2e-5 * np.abs(y).max() + 1e-6   # only the f32 summation order differs
    # either way it is the reference's arithmetic (activations quantized to int8 blocks first), not
    # dequantize-then-f32: that differs by ~5e-3
    m.close()


@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("ty,name", [(Q8_0, "q8_0"), (Q4_K, "q4_K")])
@pytest.mark.parametrize("K,M,N", [(2048, 300, 300), (4096, 1024, 1000), (512, 130, 128), (14336, 256, 257), (4096, 4096, 2048)])
def test_many_columns(oracle, K, M, N, ty, name, exact):
    """Prompt-sized batches on the tensor cores, ragged rows and columns, Q8_0 and Q4_K weights. The default kernel turns
    weights (code x block scale, for Q4_K d * sc * q - dmin * m) and activations (code x block scale of the reference's own
    Q8_0 / Q8_K quantization) into f16 operands and lets the tensor core add up all of K: two f16 roundings per product,
    within the 1e-3 bar of mul_mat, measured around 3e-4 of max|y|. TLB_PROMPT_EXACT=1 selects the kernels that keep the
    reference's integer block sums: those agree to f32 rounding."""
    import os
    rng = np.random.default_rng(K + M + N)
    W = (rng.standard_normal((M, K)) * 0.02).astype(np.float32)
    X = rng.standard_normal((N, K)).astype(np.float32)
    Wq = oracle.quantize(ty, W)
    if exact:
        os.environ["TLB_PROMPT_EXACT"] = "1"
    try:
        m, _ = mm_model(ty, K, M, N, Wq)
    finally:
        os.environ.pop("TLB_PROMPT_EXACT", None)
    (y,) = m.run(X)
    want = oracle.mul_mat(ty, Wq, K, X)
    err = close(y, want, TOL)
    print("%s [%d x %d] x %d columns, %s kernel: max error %.2e of max|y|" % (name, M, K, N, "exact" if exact else "folded-scale", err / np.abs(want).max()))
    if exact:
        assert err <= 2e-5 * np.abs(y).max() + 1e-6
    else:
        assert err <= 5e-4 * np.abs(want).max()     # half the bar: the two f16 roundings per product, not more
    m.close()


def test_config1_q8_0_4096(oracle):
    """benchmark config 1: W 4096x4096 N(0,0.02) seed 0 -> Q8_0, x N(0,1) seed 1, batch 1 and 16."""
    W = (np.random.default_rng(0).standard_normal((4096, 4096)) * 0.02).astype(np.float32)
    Wq = oracle.quantize(Q8_0, W)
    for N in (1, 16):
        X = np.random.default_rng(1).standard_normal((N, 4096)).astype(np.float32)
        m, _ = mm_model(Q8_0, 4096, 4096, N, Wq)
        (y,) = m.run(X)
        close(y, oracle.mul_mat(Q8_0, Wq, 4096, X), TOL)
        m.close()


def test_linearity_full_size(oracle):
    """Size-independent property at a benchmark shape (Q4_K 4096->14336): scaling the activations by
    a power of two scales the result exactly (quantization commutes with powers of two)."""
    rng = np.random.default_rng(11)
    W = (rng.standard_normal((14336, 4096)) * 0.02).astype(np.float32)
    from tensorlisp_b200.native import Native, quantize_rows
    n = Native(0)
    Wq = quantize_rows(n, Q4_K, W)
    n.close()
    X = rng.standard_normal((2, 4096)).astype(np.float32)
    m, _ = mm_model(Q4_K, 4096, 14336, 2, Wq)
    (y1,) = m.run(X)
    (y2,) = m.run(X * 4.0)
    assert np.array_equal(y1 * 4.0, y2)
    rows = rng.integers(0, 14336, 64)
    close(y1[:, rows], oracle.mul_mat(Q4_K, Wq[rows], 4096, X), TOL)
    m.close()


@pytest.mark.parametrize("ty", [F32, F16])
def test_plain_weights_and_batches(oracle, ty):
    """f32/f16 weights with a broadcast batch (ne2 = 2 of weights vs 4 of activations)."""
    rng = np.random.default_rng(5)
    K, M, N = 64, 10, 3
    W = rng.standard_normal((2, M, K)).astype(np.float32)
    X = rng.standard_normal((4, N, K)).astype(np.float32)
    g = G.Graph()
    w = g.weight(ty, [K, M, 2], "W")
    x = g.input(G.F32, [K, N, 4], "x")
    y = g.output(g.mul_mat(w, x))
    Wd = W.astype(np.float16) if ty == F16 else W
    m = Model(g, [Wd])
    (got,) = m.run(X)
    want = np.einsum("bmk,bnk->bnm", Wd.astype(np.float64)[[0, 0, 1, 1]], X.astype(np.float64))
    close(got.reshape(4, N, M), want, 1e-5)
    m.close()


def test_ragged_k_is_reported_by_name():
    g = G.Graph()
    w = g.weight(G.F32, [100, 4], "W")
    x = g.input(G.I32, [100, 2], "x")
    g.tensors[x].ty = G.I32
    y = g.output(g.mul_mat(w, x, "y"))
    with pytest.raises(TlbError) as e:
        Model(g, [np.zeros((4, 100), np.float32)])
    assert "MUL_MAT" in str(e.value) and "not implemented" in str(e.value)


@pytest.mark.parametrize("N", [8, 32])
def test_stream_k_schedule(oracle, N, monkeypatch):
    """A matrix of several waves of row tiles takes the stream-K schedule (equal super-block counts per
    SM, tiles cut by a CTA boundary summed by a fix-up launch); ragged last tile, and the same result as
    the tile-per-CTA schedule up to f32 summation order."""
    K, M = 512, 48000 + 37
    rng = np.random.default_rng(N)
    W = (rng.standard_normal((M, K)) * 0.02).astype(np.float32)
    X = rng.standard_normal((N, K)).astype(np.float32)
    Wq = oracle.quantize(Q4_K, W)
    m, _ = mm_model(Q4_K, K, M, N, Wq)
    (y,) = m.run(X)
    m.close()
    want = oracle.mul_mat(Q4_K, Wq, K, X)
    err = close(y, want, TOL)
    assert err <= 2e-5 * np.abs(want).max() + 1e-6
    monkeypatch.setenv("TLB_NO_STREAMK", "1")
    m, _ = mm_model(Q4_K, K, M, N, Wq)
    (y2,) = m.run(X)
    m.close()
    assert np.abs(y2 - y).max() <= 2e-5 * np.abs(want).max() + 1e-6


@pytest.mark.parametrize("K,M,N", [(256, 300, 17), (512, 130, 100), (256, 6300, 70), (1024, 2100, 400)])
def test_q4_0_beside_q8_0(oracle, K, M, N):
    """A Q4_0 and a Q8_0 matrix that read one activation: up to 64 columns they share its packed blocks, above they take different
    operands, Q4_0 in passes of 32 columns (few row tiles) or tiles of 128. Q4_0 keeps the integer sums of a block at every size, so only
    the order of K / 32 f32 additions differs: their rounding is below K / 32 * 2^-24 of the sum of the terms' magnitudes, here at most
    about sqrt(K / 32) times max|y|, 1e-5 of it at K = 1024."""
    rng = np.random.default_rng(K + M + N)
    X = rng.standard_normal((N, K)).astype(np.float32)
    Ws = [oracle.quantize(ty, (rng.standard_normal((M, K)) * 0.02).astype(np.float32)) for ty in (Q4_0, Q8_0)]
    g = G.Graph()
    w4, w8 = g.weight(Q4_0, [K, M], "W4"), g.weight(Q8_0, [K, M], "W8")
    x = g.input(G.F32, [K, N], "x")
    g.output(g.mul_mat(w4, x, "y4"))
    g.output(g.mul_mat(w8, x, "y8"))
    m = Model(g, Ws)
    y4, y8 = m.run(X)
    assert close(y4, oracle.mul_mat(Q4_0, Ws[0], K, X), TOL) <= 1e-5 * np.abs(y4).max()
    close(y8, oracle.mul_mat(Q8_0, Ws[1], K, X), TOL)
    m.close()


@pytest.mark.parametrize("N", [65, 256, 768])
@pytest.mark.parametrize("Ms", [(4096, 1024, 1024), (1024, 4096, 1024)])
def test_q4_0_matrices_of_many_and_of_few_rows_on_one_activation(oracle, Ms, N):
    """The projections of grouped-query attention. Above 64 columns a Q4_0 matrix of many rows takes tiles of 128 columns and one of few
    rows passes of 32, each with its own packing of the activation that they share (at 256 columns on 148 SMs here: 64 and 16 tiles, the line
    lies at 49). Behind a norm, as in a decoder. Integer sums of a block at every size: see test_q4_0_beside_q8_0."""
    K = 512
    rng = np.random.default_rng(N)
    X = rng.standard_normal((N, K)).astype(np.float32)
    wn = (1 + 0.1 * rng.standard_normal(K)).astype(np.float32)
    Ws = [oracle.quantize(Q4_0, (rng.standard_normal((M, K)) * 0.02).astype(np.float32)) for M in Ms]
    for normed in (False, True):
        g = G.Graph()
        tn = g.weight(G.F32, [K], "n")
        tw = [g.weight(Q4_0, [K, M], "W%d" % i) for i, M in enumerate(Ms)]
        x = g.input(G.F32, [K, N], "x")
        a = g.mul(g.rms_norm(x, 1e-5), tn) if normed else x
        for i, w in enumerate(tw):
            g.output(g.mul_mat(w, a, "y%d" % i))
        m = Model(g, [wn] + Ws)
        got = m.run(X)
        m.close()
        A = oracle.rms_norm(X, 1e-5, wn) if normed else X
        for y, w in zip(got, Ws):
            # (a norm one unit in the last place off moves a code where it lies between two)
            assert close(y, oracle.mul_mat(Q4_0, w, K, A), TOL) <= (1e-3 if normed else 1e-5) * np.abs(y).max()
