"""Products whose first operand is not a settled weight: made by the launch right in front (attention rows, keys of a rope, a cache
write, a copy into a weight leaf), kept in a state, or an input. The kernels copy weights while the launch in front is still running;
these operands have to wait for it. Every run gets other values, so that anything read early is last run's."""
import numpy as np
import pytest

from helpers import Model, close
from oracle.bindings import Q4_K, Q6_K, Q8_0
from tensorlisp_b200 import graph as G

pytestmark = pytest.mark.gpu

RUNS = 12


def product(w, x):
    return x.astype(np.float64) @ w.astype(np.float64).T


@pytest.mark.parametrize("n", [1, 9])
@pytest.mark.parametrize("seqs,ctx", [(96, 64), (40, 700)])
def test_rows_of_an_attention(n, seqs, ctx):
    hs, heads, kvh, bs = 128, 16, 4, 16
    rng = np.random.default_rng(seqs + n)
    blocks = (ctx + bs - 1) // bs
    pool = seqs * blocks * kvh * bs * hs
    g = G.Graph()
    kc, vc = g.state(G.F16, [pool], "k"), g.state(G.F16, [pool], "v")
    q, x = g.input(G.F32, [hs, heads, seqs], "q"), g.input(G.F32, [hs, n], "x")
    tables, lens = g.input(G.I32, [blocks, seqs], "tables"), g.input(G.I32, [seqs], "lens")
    a = g.output(g.paged_attention(g.cast(q, G.F16), kc, vc, tables, lens, bs, ctx, hs ** -0.5, kvh))
    y = g.output(g.mul_mat(g.reshape(a, [hs, heads * seqs]), x, "y"))
    m = Model(g, [], [2 * pool] * 2, [("y", y), ("a", a)])
    for off in m.native.state_offsets:
        m.native.state.write(off, rng.standard_normal(pool, np.float32).astype(np.float16))
    table = rng.permutation(seqs * blocks).astype(np.int32).reshape(seqs, blocks)
    for _ in range(RUNS):
        Q, X = 3 * rng.standard_normal((seqs, heads, hs)).astype(np.float32), rng.standard_normal((n, hs)).astype(np.float32)
        got, rows = m.run(Q, X, table, rng.integers(1, ctx + 1, seqs).astype(np.int32))
        close(got.reshape(n, -1), product(rows.reshape(-1, hs), X), 1e-5)
    m.close()


@pytest.mark.parametrize("what", ["keys of the prompt", "the pool of the prompt", "the pool of a decode step"])
def test_keys_that_a_rope_writes(what):
    hs, heads, kvh, bs, T, n = 64, 4, 2, 16, 512, 3
    rng = np.random.default_rng(len(what))
    g = G.Graph()
    pool = T * kvh * hs
    kc, vc = g.state(G.F16, [pool], "kc"), g.state(G.F16, [pool], "vc")
    qkv = [g.input(G.F32, [h * hs, T], s) for h, s in ((heads, "q"), (kvh, "k"), (kvh, "v"))]
    pos, slots, x = g.input(G.I32, [T], "pos"), g.input(G.I32, [2 * T], "slots"), g.input(G.F32, [hs, n], "x")
    rope = lambda t, h: g.rope_ext(g.reshape(t, [hs, h, T]), pos, None, hs, 2, 0, 10000.0, 1.0, 0.0, 1.0, 0.0, 0.0)
    qr, kr = rope(qkv[0], heads), rope(qkv[1], kvh)
    k16, v16 = g.cast(g.reshape(kr, [hs * kvh, T]), G.F16), g.cast(qkv[2], G.F16)
    g.paged_cache_write(k16, v16, kc, vc, slots, bs, kvh)
    if what == "keys of the prompt":
        y = g.mul_mat(g.view(k16, [hs, T], hs * kvh * 2), x, "y")                # keys of head 0
    else:
        y = g.mul_mat(g.view(kc, [hs, T * kvh], hs * 2), x, "y")
    outs = [("y", g.output(y))]
    extra = []
    if what == "the pool of a decode step":
        tables, lens = g.input(G.I32, [1, T], "tables"), g.input(G.I32, [T], "lens")
        extra = [np.arange(T, dtype=np.int32) // bs, np.ones(T, np.int32)]
        g.output(g.cast(g.paged_attention(g.cast(qr, G.F16), kc, vc, tables, lens, bs, bs, 1.0, kvh), G.F32))
    else:
        kv, vv = (g.permute(g.reshape(t, [hs, kvh, T, 1]), 0, 2, 1, 3) for t in (k16, v16))
        g.output(g.flash_attn_ext(g.permute(g.reshape(qr, [hs, heads, T, 1]), 0, 2, 1, 3), kv, vv, None, 0.125))
    outs.append(("keys", g.output(g.cast(k16, G.F32))))
    m = Model(g, [], [2 * pool] * 2, outs)
    for run in range(RUNS):
        ins = [rng.standard_normal((T, h * hs)).astype(np.float32) for h in (heads, kvh, kvh)]
        X = rng.standard_normal((n, hs)).astype(np.float32)
        where = rng.permutation(T).astype(np.int64)
        got, keys = m.run(*ins, rng.integers(0, 1000, T).astype(np.int32), where.view(np.int32), X, *extra)
        keys = keys.reshape(T, kvh, hs)
        if what == "keys of the prompt":
            rows = keys[:, 0]
        else:                                       # pool: [block][head][token of the block][hs]
            rows = np.zeros((T // bs, kvh, bs, hs), np.float32)
            rows[where // bs, :, where % bs] = keys
            rows = rows.reshape(-1, hs)
        close(got.reshape(n, -1), product(rows, X), 1e-5)
    m.close()


def test_a_weight_leaf_that_the_program_writes():
    k, rows, n = 256, 4096, 2
    rng = np.random.default_rng(0)
    g = G.Graph()
    w, new, x = g.weight(G.F16, [k, rows], "W"), g.input(G.F32, [k, rows], "new"), g.input(G.F32, [k, n], "x")
    g.cpy(new, w)
    y = g.output(g.mul_mat(w, x, "y"))
    m = Model(g, [np.zeros((rows, k), np.float16)], [], [("y", y)])
    for _ in range(RUNS):
        W, X = rng.standard_normal((rows, k)).astype(np.float16), rng.standard_normal((n, k)).astype(np.float32)
        (got,) = m.run(W.astype(np.float32), X)
        close(got.reshape(n, rows), product(W, X), 1e-5)
    m.close()


@pytest.mark.parametrize("ty", [Q8_0, Q4_K, Q6_K])
@pytest.mark.parametrize("n", [1, 20, 300])
@pytest.mark.parametrize("kind", ["state", "input"])
def test_quantized_operands_that_are_no_weights(oracle, ty, n, kind):
    k, rows = 512, 200
    rng = np.random.default_rng(n)
    g = G.Graph()
    w = g.state(ty, [k, rows], "W") if kind == "state" else g.input(ty, [k, rows], "W")
    x = g.input(G.F32, [k, n], "x")
    y = g.output(g.mul_mat(w, x, "y"))
    size = k * rows // G.TYPE_TRAITS[ty][1] * G.TYPE_TRAITS[ty][2]
    m = Model(g, [], [size] if kind == "state" else [], [("y", y)])
    for _ in range(3):
        X = rng.standard_normal((n, k)).astype(np.float32)
        Wq = oracle.quantize(ty, (rng.standard_normal((rows, k)) * 0.02).astype(np.float32))
        if kind == "state":
            m.native.state.write(m.native.state_offsets[0], Wq)
            (got,) = m.run(X)
        else:
            (got,) = m.run(Wq, X)
        want = product(oracle.dequantize(ty, Wq, k).reshape(rows, k), X) if ty == Q6_K else oracle.mul_mat(ty, Wq, k, X)
        # 300 columns of Q8_0 / Q4_K: f16 operands with the scales folded in, 3e-4 of the largest result at most
        close(got.reshape(n, rows), want, 5e-4 if n == 300 else 2e-5)
    m.close()
