"""A node that is folded into a later launch is read there: the values it reads must be those of its own place in the graph. Every
graph here writes new values over a source of the folded node between the two (a state that a program updates in place), at the
column counts of the three routes a product takes; the oracle works on the old values."""
import numpy as np
import pytest

from helpers import Model, close
from oracle.bindings import Q4_0, Q4_K, Q8_0
from tensorlisp_b200 import graph as G

pytestmark = pytest.mark.gpu

K, M = 512, 96
CASES = ["cast", "norm", "norm_late", "norm_weight", "norm_through_a_view", "add_first", "add_second", "add_then_set_rows", "gate", "up", "silu_late"]


def build(case, g, N, S, ws, oracle, X, Y, NEW):
    """The activation's node and its values. S: f32 state [K, N] holding X; `new` is copied over it behind the reads."""
    x, new = g.input(G.F32, [K, N], "x"), g.input(G.F32, [K, N], "new")
    norm = g.weight(G.F32, [K], "norm")
    overwrite = lambda dst=S: g.cpy(new, dst)
    if case == "cast":
        H = g.state(G.F16, [K, N], "half")          # zeros, and what the first run leaves behind
        g.cpy(x, H)
        c = g.cast(H, G.F32)
        g.cpy(new, H)
        return c, Y.astype(np.float16).astype(np.float32)
    if case in ("norm", "norm_through_a_view"):
        src = S if case == "norm" else g.view(S, [K, N], K * 4, name="view")
        t = g.mul(g.rms_norm(src, 1e-5), norm)
        overwrite()
        return t, oracle.rms_norm(X, 1e-5, ws[0])
    if case == "norm_late":
        n = g.rms_norm(S, 1e-5)
        overwrite()
        return g.mul(n, norm), oracle.rms_norm(X, 1e-5, ws[0])
    if case == "norm_weight":
        row = g.view(S, [K], name="row0")
        t = g.mul(g.rms_norm(x, 1e-5), row)
        overwrite()
        return t, oracle.rms_norm(Y, 1e-5, np.ascontiguousarray(X[0]))
    if case in ("add_first", "add_second"):
        h = g.add(S, x) if case == "add_first" else g.add(x, S)
        t = g.mul(g.rms_norm(h, 1e-5), norm)
        overwrite()
        return t, oracle.rms_norm(X + Y, 1e-5, ws[0])
    if case == "add_then_set_rows":
        h = g.add(S, x)
        t = g.mul(g.rms_norm(h, 1e-5), norm)
        first = g.input(G.I32, [1], "first")
        g.output(g.set_rows(h, g.view(new, [K, 1], K * 4), first))     # row 0 of the sum becomes row 0 of `new`
        return t, oracle.rms_norm(X + Y, 1e-5, ws[0])
    if case in ("gate", "up"):
        a = g.glu(S, b=x) if case == "gate" else g.glu(x, b=S)
        overwrite()
        return a, oracle.silu_mul(X, Y) if case == "gate" else oracle.silu_mul(Y, X)
    if case == "silu_late":
        s = g.silu(S)
        overwrite()
        return g.mul(s, x), oracle.silu_mul(X, Y)


@pytest.mark.parametrize("ty,N", [(Q8_0, 1), (Q4_0, 2), (Q4_K, 1), (Q4_K, 2), (Q4_K, 5), (Q4_K, 40), (Q8_0, 6), (Q8_0, 300)])
@pytest.mark.parametrize("case", CASES)
def test_sources_keep_their_place(oracle, case, ty, N):
    rng = np.random.default_rng(N + len(case))
    X, Y, NEW = rng.standard_normal((3, N, K)).astype(np.float32)
    W = oracle.quantize(ty, (rng.standard_normal((M, K)) * 0.02).astype(np.float32))
    wn = (1 + 0.1 * rng.standard_normal(K)).astype(np.float32)
    g = G.Graph()
    S = g.state(G.F32, [K, N], "S")
    t, T = build(case, g, N, S, [wn], oracle, X, Y, NEW)
    y = g.output(g.mul_mat(g.weight(ty, [K, M], "W"), t, "y"))
    m = Model(g, [wn, W], [4 * K * N] + ([2 * K * N] if case == "cast" else []), [("y", y)])
    for _ in range(2):
        m.native.state.write(m.native.state_offsets[0], X)
        (got,) = m.run(*((Y, NEW) + ((np.zeros(1, np.int32),) if case == "add_then_set_rows" else ())))
        close(got.reshape(N, M), oracle.mul_mat(ty, W, K, T), 2e-3)
    if case == "add_then_set_rows":
        h = m.program.read(g.keep[0]).reshape(N, K)
        assert np.array_equal(h[0], NEW[0]) and np.array_equal(h[1:], (X + Y)[1:])
    m.close()


@pytest.mark.parametrize("prompt", [False, True])
def test_rope_reads_its_queries_keys_and_values_in_place(oracle, prompt):
    """The ropes, casts and the cache write of a layer become one launch at the cache write's place."""
    hd, heads, kvh, bs, n = 64, 4, 2, 16, 24
    rng = np.random.default_rng(5)
    q, k, v = (rng.standard_normal((n, h * hd)).astype(np.float32) for h in (heads, kvh, kvh))
    junk = rng.standard_normal((n, heads * hd)).astype(np.float32)
    outs = []
    for write in ("", "q", "k", "v", "pos"):
        g = G.Graph()
        pool = 2 * bs * kvh * hd
        kc, vc = g.state(G.F16, [pool], "kc"), g.state(G.F16, [pool], "vc")
        sq, sk, sv = (g.state(G.F32, [h * hd, n], s) for h, s in ((heads, "q"), (kvh, "k"), (kvh, "v")))
        sp = g.state(G.I32, [n], "pos")
        new, slots = g.input(G.F32, [heads * hd, n], "junk"), g.input(G.I32, [2 * n], "slots")
        rope = lambda t: g.rope_ext(t, sp, None, hd, 2, 0, 10000.0, 1.0, 0.0, 1.0, 0.0, 0.0)
        qr = rope(g.reshape(sq, [hd, heads, n]))
        kr = rope(g.reshape(sk, [hd, kvh, n]))
        k16, v16 = g.cast(g.reshape(kr, [hd * kvh, n]), G.F16), g.cast(sv, G.F16)
        if write == "q":
            g.cpy(new, sq)
        elif write == "k":
            g.cpy(g.view(new, [kvh * hd, n], heads * hd * 4), sk)
        elif write == "v":
            g.cpy(g.view(new, [kvh * hd, n], heads * hd * 4), sv)
        elif write == "pos":
            g.cpy(g.cast(g.view(new, [n]), G.I32), sp)
        g.paged_cache_write(k16, v16, kc, vc, slots, bs, kvh)
        if prompt:
            qv = g.permute(g.reshape(qr, [hd, heads, n, 1]), 0, 2, 1, 3)
            kv, vv = (g.permute(g.reshape(t, [hd, kvh, n, 1]), 0, 2, 1, 3) for t in (k16, v16))
            out = g.output(g.flash_attn_ext(qv, kv, vv, None, hd ** -0.5))
        else:
            tables, lens = g.input(G.I32, [2, n], "tables"), g.input(G.I32, [n], "lens")
            out = g.output(g.cast(g.paged_attention(g.cast(qr, G.F16), kc, vc, tables, lens, bs, 2 * bs, hd ** -0.5, kvh), G.F32))
        m = Model(g, [], [2 * pool] * 2 + [q.nbytes, k.nbytes, v.nbytes, 4 * n], [("out", out)])
        for off, a in zip(m.native.state_offsets[2:], (q, k, v, np.arange(n, dtype=np.int32))):
            m.native.state.write(off, a)
        ins = [junk, np.arange(n, dtype=np.int64).view(np.int32)]
        if not prompt:
            ins += [np.tile(np.arange(2, dtype=np.int32), n), np.arange(1, n + 1, dtype=np.int32)]
        outs.append(m.run(*ins)[0].copy())
        m.close()
    for write, o in zip("q k v pos".split(), outs[1:]):
        close(o, outs[0], 1e-6)
