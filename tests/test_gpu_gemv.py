"""The few-column mul_mat kernels at the edges of their tiles: row groups of 16, row segments of four or eight super-blocks,
one to eight columns per launch (Q6_K: one to four), short rows that share a tile, and the nodes folded into a launch."""
import numpy as np
import pytest

from helpers import Model, close
from oracle.bindings import Q4_0, Q4_K, Q6_K, Q8_0
from tensorlisp_b200 import graph as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ty", [Q4_K, Q8_0, Q4_0, Q6_K])
@pytest.mark.parametrize("K,M,N", [(256, 1, 1), (256, 2385, 3), (512, 17, 2), (768, 333, 5), (1280, 2369, 1), (2304, 31, 8), (2304, 148 * 16 + 9, 2), (4096, 130, 9), (16384, 40, 4),
                                   (28672, 65, 7), (1024, 40001, 1)])
def test_edges(oracle, ty, K, M, N):
    rng = np.random.default_rng(K + M + N)
    W = (rng.standard_normal((M, K)) * 0.02).astype(np.float32)
    X = (rng.standard_normal((N, K)) * np.exp(rng.standard_normal((N, 1)) * 3)).astype(np.float32)
    X[0, :300] = 0
    Wq = oracle.quantize(ty, W)
    g = G.Graph()
    g.output(g.mul_mat(g.weight(ty, [K, M], "W"), g.input(G.F32, [K, N], "x"), "y"))
    m = Model(g, [Wq])
    want = X.astype(np.float64) @ oracle.dequantize(ty, Wq, K).reshape(M, K).astype(np.float64).T if ty == Q6_K else oracle.mul_mat(ty, Wq, K, X)
    for _ in range(2):   # (the second run finds the first one's stages in shared memory)
        (got,) = m.run(X)
        for n in range(N):
            close(got.reshape(N, M)[n], want.reshape(N, M)[n], 2e-5)
    m.close()


@pytest.mark.parametrize("ty", [Q4_K, Q8_0, Q4_0])
@pytest.mark.parametrize("d,f,n", [(512, 768, 1), (768, 512, 2), (512, 2560, 3), (2048, 4864, 1), (8448, 256, 2)])
def test_folded_nodes(oracle, ty, d, f, n):
    """Residual add, norm, gate and up, SiLU(gate) * up, f16 cast in front of a product: what the launches take in."""
    rng = np.random.default_rng(d + f + n)
    mk = lambda k, m: (rng.standard_normal((m, k)) * 0.02).astype(np.float32)
    ws = [oracle.quantize(ty, mk(k, m)) for k, m in ((d, f), (d, f), (f, d), (d, 96), (d, 40), (d, 24))]
    wn = (1 + 0.1 * rng.standard_normal(d)).astype(np.float32)
    g = G.Graph()
    x, r = g.input(G.F32, [d, n], "x"), g.input(G.F32, [d, n], "r")
    norm = g.weight(G.F32, [d], "norm")
    gate, up, down, q, k, v = [g.weight(ty, [a, b], s) for s, a, b in (("gate", d, f), ("up", d, f), ("down", f, d), ("q", d, 96), ("k", d, 40), ("v", d, 24))]
    h = g.add(x, r, "h")
    t = g.mul(g.rms_norm(h, 1e-5), norm, "t")
    y = g.mul_mat(down, g.glu(g.mul_mat(gate, t, "g"), b=g.mul_mat(up, t, "u"), name="a"), "y")
    o = g.output(g.add(h, y, "o"))
    c = g.cast(g.cast(o, G.F16), G.F32)
    outs = [g.output(g.mul_mat(w, c, s)) for w, s in ((q, "yq"), (k, "yk"), (v, "yv"))]
    m = Model(g, [wn] + ws)
    X, R = rng.standard_normal((2, n, d)).astype(np.float32)
    got = m.run(X, R)
    H = X + R
    T = oracle.rms_norm(H, 1e-5, wn)
    O = H + oracle.mul_mat(ty, ws[2], f, oracle.silu_mul(oracle.mul_mat(ty, ws[0], d, T), oracle.mul_mat(ty, ws[1], d, T)))
    close(got[0].reshape(n, d), O, 1e-3)
    C = got[0].reshape(n, d).astype(np.float16).astype(np.float32)
    for y, w in zip(got[1:], ws[3:]):
        close(y.reshape(n, -1), oracle.mul_mat(ty, w, d, C), 2e-5)
    m.close()


@pytest.mark.parametrize("K,M,N", [(28672, 3601, 3), (256, 488289, 4), (4096, 54945, 8)])
def test_several_columns_of_a_long_stream(oracle, K, M, N):
    """Q4_K from three columns on: the smallest matrices that few_column_faster leaves to this kernel."""
    rng = np.random.default_rng(K + M + N)
    assert 25_000_000 * (N + 1) <= K * M < 26_000_000 * (N + 1)
    from tensorlisp_b200.native import Native, quantize_rows
    native = Native(0)
    Wq = quantize_rows(native, Q4_K, (rng.standard_normal((M, K), np.float32) * np.float32(0.02)))
    native.close()
    X = rng.standard_normal((N, K)).astype(np.float32)
    g = G.Graph()
    g.output(g.mul_mat(g.weight(Q4_K, [K, M], "W"), g.input(G.F32, [K, N], "x"), "y"))
    m = Model(g, [Wq])
    (got,) = m.run(X)
    rows = np.unique(np.concatenate([[0, 15, 16, M - 1], rng.integers(0, M, 400)]))
    close(got.reshape(N, M)[:, rows], oracle.mul_mat(Q4_K, np.ascontiguousarray(Wq.reshape(M, -1)[rows]), K, X), 2e-5)
    m.close()


def folded_block(ty, d, f, n, ws, wn):
    g = G.Graph()
    x, r = g.input(G.F32, [d, n], "x"), g.input(G.F32, [d, n], "r")
    norm = g.weight(G.F32, [d], "norm")
    gate, up, down, q, k, v = [g.weight(ty, [a, b], s) for s, a, b in (("gate", d, f), ("up", d, f), ("down", f, d), ("q", d, 96), ("k", d, 40), ("v", d, 24))]
    h = g.add(x, r, "h")
    t = g.mul(g.rms_norm(h, 1e-5), norm, "t")
    y = g.mul_mat(down, g.glu(g.mul_mat(gate, t, "g"), b=g.mul_mat(up, t, "u"), name="a"), "y")
    o = g.output(g.add(h, y, "o"))
    c = g.cast(g.cast(o, G.F16), G.F32)
    for w, s in ((q, "yq"), (k, "yk"), (v, "yv")):
        g.output(g.mul_mat(w, c, s))
    return Model(g, [wn] + ws)


@pytest.mark.parametrize("ty", [Q4_K, Q8_0, Q4_0])
@pytest.mark.parametrize("d,f", [(512, 768), (2048, 4864), (8448, 256), (4096, 2560)])
def test_rows_quantized_in_the_launch_or_in_front_of_it(oracle, monkeypatch, ty, d, f):
    """One and two columns produce and quantize their rows in the product's own launch, three get them from the row quantizers; the rows
    they share come out the same to the last bit."""
    rng = np.random.default_rng(d + f)
    mk = lambda k, m: (rng.standard_normal((m, k)) * 0.02).astype(np.float32)
    ws = [oracle.quantize(ty, mk(k, m)) for k, m in ((d, f), (d, f), (f, d), (d, 96), (d, 40), (d, 24))]
    wn = (1 + 0.1 * rng.standard_normal(d)).astype(np.float32)
    X, R = rng.standard_normal((2, 3, d)).astype(np.float32)
    monkeypatch.setenv("TLB_NO_TC", "1")        # three columns stay on this kernel
    seen = []
    for n in (3, 1, 2):
        m = folded_block(ty, d, f, n, ws, wn)
        seen.append((n, m.program.dispatch_count(), [a.reshape(n, -1).copy() for a in m.run(X[:n], R[:n])]))
        m.close()
    assert seen[1][1] == seen[2][1] == 5 < seen[0][1]
    for n, _, got in seen[1:]:
        for a, b in zip(got, seen[0][2]):
            assert a.tobytes() == b[:n].tobytes()


# The Q6_K tests from here on run twice: with the kernel that a size takes, and with TLB_Q6_DIGITS, which sends matrices below the lines of gemv_q6_columns
# and mm_q6_supported to the kernels behind them, too, so that their edges need no large matrices.
def pytest_generate_tests(metafunc):
    if metafunc.function.__name__.startswith("test_q6_K"):
        metafunc.fixturenames.append("q6_route")
        metafunc.parametrize("q6_route", ["by size", "digits"], indirect=True)


@pytest.fixture
def q6_route(request, monkeypatch):
    if request.param == "digits":
        monkeypatch.setenv("TLB_Q6_DIGITS", "1")


@pytest.mark.parametrize("K,M", [(256, 130), (768, 45), (1792, 300), (2048, 17), (4096, 148 * 32 + 5), (7168, 33), (7424, 40), (14336, 20)])
def test_q6_K_against_f64(oracle, K, M):
    """Activations as eight digits of eight bits: rows of less than eight super-blocks (several row groups per tile), whole rows, segments of eight, one to four
    columns of rows that have as many; and 7424 (29 super-blocks), whose rows do not fit and take the kernel that decodes, like the further columns of
    longer rows. Whole numbers are exact, so the error is that of one f32 sum over the super-blocks and the eight warps: a few units in the last place of
    the result's root mean square, whatever the spread of the values."""
    rng = np.random.default_rng(K + M)
    Wq = oracle.quantize(Q6_K, (rng.standard_normal((M, K)) * 0.02).astype(np.float32))
    W = oracle.dequantize(Q6_K, Wq, K).reshape(M, K).astype(np.float64)
    for N in (1, 2, 3, 4, 7):
        X = (rng.standard_normal((N, K)) * np.exp(2 * rng.standard_normal((N, K)))).astype(np.float32)
        g = G.Graph()
        g.output(g.mul_mat(g.weight(Q6_K, [K, M], "W"), g.input(G.F32, [K, N], "x"), "y"))
        m = Model(g, [Wq])
        for scale in (1.0, 2.0 ** 60, 2.0 ** -80):
            (got,) = m.run((X * np.float32(scale)).astype(np.float32))
            want = (X * np.float32(scale)).astype(np.float64) @ W.T
            assert np.linalg.norm(got.reshape(N, M) - want) <= 2.5e-7 * np.linalg.norm(want)
        m.close()


@pytest.mark.parametrize("N", [1, 2])
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_q6_K_values_that_are_not_finite(oracle, bad, N):
    rng = np.random.default_rng(N)
    K, M = 4096, 64
    Wq = oracle.quantize(Q6_K, (rng.standard_normal((M, K)) * 0.02).astype(np.float32))
    X = rng.standard_normal((N, K)).astype(np.float32)
    X[0, 777] = bad
    g = G.Graph()
    g.output(g.mul_mat(g.weight(Q6_K, [K, M], "W"), g.input(G.F32, [K, N], "x"), "y"))
    m = Model(g, [Wq])
    (got,) = m.run(X)
    with np.errstate(invalid="ignore"):
        want = X.astype(np.float64) @ oracle.dequantize(Q6_K, Wq, K).reshape(M, K).astype(np.float64).T
    got = got.reshape(N, M)
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isinf(got), np.isinf(want))
    inf, fin = np.isinf(want), np.isfinite(want)
    assert np.array_equal(np.sign(got[inf]), np.sign(want[inf])) and np.allclose(got[fin], want[fin], atol=1e-5)
    m.close()


@pytest.mark.parametrize("N", [1, 2, 3, 4, 7])
@pytest.mark.parametrize("K", [768, 2048])
def test_q6_K_several_values_that_are_not_finite(oracle, K, N):
    """Infinities of either sign side by side in a super-block, in two of them and over weights of zero (infinite, or undefined where they cancel or meet
    a zero), and a row whose scale is infinite: the same kind of value as the sum of products, whichever kernel the columns take."""
    rng = np.random.default_rng(K + N)
    M = 170
    Wq = oracle.quantize(Q6_K, (rng.standard_normal((M, K)) * 0.02).astype(np.float32)).copy()
    blocks = Wq.view(np.uint8).reshape(M, K // 256, 210)
    blocks[5, 1, 208:210] = np.frombuffer(np.float16(np.inf).tobytes(), np.uint8)
    blocks[9, 0, :64] = blocks[9, 0, 128:160] = 0      # codes of 0 (a weight of -32 d sc) ...
    blocks[10, 0, 192:200] = 0                         # ... and scales of 0
    W = oracle.dequantize(Q6_K, Wq, K).reshape(M, K).astype(np.float64)
    g = G.Graph()
    g.output(g.mul_mat(g.weight(Q6_K, [K, M], "W"), g.input(G.F32, [K, N], "x"), "y"))
    m = Model(g, [Wq])
    for places in ([3, 70], [3, 4, 130], [7, 300], [255, 256, 600], [0, 1, 2, 3, 127, 511]):
        for signs in ("++++++", "------", "+-+-+-"):
            X = rng.standard_normal((N, K)).astype(np.float32)
            for at, s in zip(places, signs):
                X[N - 1, at] = np.inf if s == "+" else -np.inf
            (got,) = m.run(X)
            with np.errstate(invalid="ignore"):
                want = np.stack([(W * x).sum(1) for x in X.astype(np.float64)])
            got = got.reshape(N, M)
            assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isinf(got), np.isinf(want))
            inf, fin = np.isinf(want), np.isfinite(want)
            assert np.array_equal(np.sign(got[inf]), np.sign(want[inf])) and np.allclose(got[fin], want[fin], atol=1e-5)
    m.close()


def outlier_rows(oracle, N, large, K=2048, M=150):
    """Every row has weights of zero where a column's large values are; row sums in f64 and the norms of the rows' other terms."""
    rng = np.random.default_rng(N)
    W = (rng.standard_normal((M, K)) * 0.02).astype(np.float32)
    at = rng.choice(K, 12, replace=False)
    W[:, at] = 0
    X = rng.standard_normal((N, K)).astype(np.float32)
    X[:, at] = (large * (1 + rng.random((N, 12)))).astype(np.float32)
    Wq = oracle.quantize(Q6_K, W)
    W = oracle.dequantize(Q6_K, Wq, K).reshape(M, K).astype(np.float64)
    assert not W[:, at].any()
    terms = X.astype(np.float64)[:, None, :] * W
    g = G.Graph()
    g.output(g.mul_mat(g.weight(Q6_K, [K, M], "W"), g.input(G.F32, [K, N], "x"), "y"))
    m = Model(g, [Wq])
    (got,) = m.run(X)
    m.close()
    return np.abs(got.reshape(N, M) - terms.sum(-1)), np.sqrt((terms ** 2).sum(-1))


@pytest.mark.parametrize("large", [1e0, 1e2, 1e4, 1e6, 1e8, 1e15, 1e30])
@pytest.mark.parametrize("N", [1, 2, 3, 5, 13])
def test_q6_K_large_values_over_weights_of_zero(oracle, N, large):
    """Large activations under zero codes take no bits from the rest of their super-block. Row by row: the whole-number sums of a super-block are exact and get
    four roundings, one more each as they and eight warps' parts are added up. Decoded, a lane adds 16 terms (value by value) or 64 in four sums, and a
    warp's 32 lanes: about 40 roundings that a result goes through, of partial sums that stay below the norm of all terms for random signs. At 2^-24 of
    that at most each and of random sign, three standard deviations are 3 x sqrt(40 / 3) = 11 of them."""
    off, norm = outlier_rows(oracle, N, large)
    assert (off <= 11 * 2.0 ** -24 * norm).all(), (off / norm).max()


@pytest.mark.parametrize("N,K", [(1, 1280), (2, 1280), (3, 1280), (4, 768), (5, 1280), (13, 1280)])
def test_q6_K_single_terms(oracle, N, K):
    """A row with one weight: the product of that weight and its activation to a few roundings (four with digits, three value by value, one in the bound for
    both), however small the activation is beside the others of its super-block."""
    rng = np.random.default_rng(N)
    M = 900
    W = np.zeros((M, K), np.float32)
    at = rng.integers(0, K, M)
    W[np.arange(M), at] = rng.standard_normal(M)
    Wq = oracle.quantize(Q6_K, W)
    W = oracle.dequantize(Q6_K, Wq, K).reshape(M, K).astype(np.float64)
    g = G.Graph()
    g.output(g.mul_mat(g.weight(Q6_K, [K, M], "W"), g.input(G.F32, [K, N], "x"), "y"))
    m = Model(g, [Wq])
    for spread in (1, 4, 12):
        X = (rng.standard_normal((N, K)) * np.exp(spread * rng.standard_normal((N, K)))).astype(np.float32)
        (got,) = m.run(X)
        want = X.astype(np.float64) @ W.T
        assert np.all(np.abs(got.reshape(N, M) - want) <= 5 * 2.0 ** -24 * np.abs(want))
    m.close()


@pytest.mark.parametrize("K,M,N", [(256, 8, 5), (512, 9, 6), (768, 135, 16), (4096, 1500, 17), (1024, 7, 12), (2048, 148 * 128 + 3, 9), (14336, 40, 22), (256, 130, 64), (4096, 20000, 21)])
def test_q6_K_on_the_tensor_cores(oracle, K, M, N):
    """The kernel of three columns and more: rows in eights and what is left of them (fewer than eight rows stay with the other kernel), tiles cut between CTAs and
    whole, several passes of columns. The sums of a super-block are exact, so the error is that of some eight roundings per super-block and of the
    addition of a tile's parts: below 2.5e-7 of the result's norm. (Row by row: test_q6_K_large_values_over_weights_of_zero.)"""
    rng = np.random.default_rng(K + M + N)
    Wq = oracle.quantize(Q6_K, (rng.standard_normal((M, K)) * 0.02).astype(np.float32))
    W = oracle.dequantize(Q6_K, Wq, K).reshape(M, K).astype(np.float64)
    X = rng.standard_normal((N, K)).astype(np.float32)
    X[1, :256] = 0.0
    g = G.Graph()
    g.output(g.mul_mat(g.weight(Q6_K, [K, M], "W"), g.input(G.F32, [K, N], "x"), "y"))
    m = Model(g, [Wq])
    for scale in (1.0, 2.0 ** 100, 2.0 ** -60):
        (got,) = m.run((X * np.float32(scale)).astype(np.float32))
        want = (X * np.float32(scale)).astype(np.float64) @ W.T
        assert np.linalg.norm(got.reshape(N, M) - want) <= 2.5e-7 * np.linalg.norm(want)
    m.close()


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan, 1e-39])
def test_q6_K_on_the_tensor_cores_unusual_values(oracle, bad):
    """An infinite, undefined or denormal activation, and a row whose scale is infinite, where the digits cannot hold them."""
    rng = np.random.default_rng(5)
    K, M, N = 2048, 140, 7
    Wq = oracle.quantize(Q6_K, (rng.standard_normal((M, K)) * 0.02).astype(np.float32)).copy()
    rows = Wq.view(np.uint8).reshape(M, K // 256, 210)
    rows[3, 2, 208:210] = np.frombuffer(np.float16(np.inf).tobytes(), np.uint8)
    X = rng.standard_normal((N, K)).astype(np.float32)
    if np.isfinite(bad):
        X[2, 512:768] = bad * X[2, 512:768]   # a whole block of such values
    else:
        X[2, 777] = bad
    g = G.Graph()
    g.output(g.mul_mat(g.weight(Q6_K, [K, M], "W"), g.input(G.F32, [K, N], "x"), "y"))
    m = Model(g, [Wq])
    (got,) = m.run(X)
    with np.errstate(invalid="ignore"):
        want = X.astype(np.float64) @ oracle.dequantize(Q6_K, Wq, K).reshape(M, K).astype(np.float64).T
    got = got.reshape(N, M)
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isinf(got), np.isinf(want))
    fin = np.isfinite(want)
    assert np.allclose(got[fin], want[fin], atol=1e-5)
    m.close()


@pytest.mark.parametrize("N", [1, 2, 3])
@pytest.mark.parametrize("K", [2048, 1792])
def test_q6_K_matrices_on_one_activation(oracle, K, N):
    """Projections of one activation, and gate and up in front of a gated product, with rows that are a multiple of 16 bytes (2048 weights) and that
    are not: the few-column kernels of the other types take such matrices in one launch, the Q6_K ones take one each. Bound as in
    test_q6_K_against_f64; the gate adds the exponential's and the division's two units in the last place, the second product's input rounding none (f32)."""
    rng = np.random.default_rng(K + N)
    X = rng.standard_normal((N, K)).astype(np.float32)
    Ws = [oracle.quantize(Q6_K, (rng.standard_normal((M, K)) * 0.02).astype(np.float32)) for M in (512, 128, 512)]
    D = [oracle.dequantize(Q6_K, w, K).reshape(-1, K).astype(np.float64) for w in Ws]
    g = G.Graph()
    x = g.input(G.F32, [K, N], "x")
    ys = [g.mul_mat(g.weight(Q6_K, [K, len(d)], "W%d" % i), x, "y%d" % i) for i, d in enumerate(D)]
    for y in ys:
        g.output(y)
    gate, up = (g.mul_mat(g.weight(Q6_K, [K, 512], n), x, n) for n in ("gate", "up"))
    g.output(g.mul(g.silu(gate), up))
    m = Model(g, Ws + [Ws[0], Ws[2]])
    *got, h = m.run(X)
    m.close()
    want = [X.astype(np.float64) @ d.T for d in D]
    for a, b in zip(got, want):
        assert np.linalg.norm(a.reshape(b.shape) - b) <= 2.5e-7 * np.linalg.norm(b)
    b = want[0] / (1 + np.exp(-want[0])) * want[2]
    assert np.linalg.norm(h.reshape(b.shape) - b) <= 1e-6 * np.linalg.norm(b)
