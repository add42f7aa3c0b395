"""End-to-end parity of the SwiGLU FFN block (benchmark config 2) and of a whole decode step of a
Llama-shaped decoder (benchmark config 4 geometry at reduced depth / width / vocabulary) against the
oracle.

Two kinds of check on the decode step:
 * teacher-forced, op by op: every tapped intermediate of the GPU run is compared with the oracle
   applied to the GPU's OWN inputs of that op. Bars: mul_mat / attention 1e-3 of max|want|, row ops 1e-5.
 * end to end: logits against the oracle run from the token ids. The reference's arithmetic
   re-quantizes activations to int8 before every mul_mat, which makes the logits a discontinuous
   function of the inputs: the oracle's own logits move by 1e-2..1e-1 when its mul_mat outputs are
   perturbed by 1e-6 relative (the size of an f32 summation-order difference), because one flipped
   code is amplified by the RMS norms of an N(0, 0.02)-initialised residual stream. The end-to-end
   bar is therefore max(1e-2, the oracle's measured 1e-6-noise envelope), with identical top-1
   wherever the oracle's own top-1 margin exceeds that envelope.
"""
import copy

import numpy as np
import pytest

from helpers import Model, NoisyOracle, close, make_decoder_weights, oracle_decoder_step
from oracle.bindings import Q4_K, Q8_0
from tensorlisp_b200 import graph as G
from tensorlisp_b200.programs import DecoderConfig, decoder_step, swiglu_ffn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 32])
def test_ffn_block_config2(oracle, T):
    """RMSNorm(eps 1e-5, w ~ N(1, 0.1)) -> gate/up 4096->14336 Q4_K -> SiLU(gate)*up -> down 14336->4096."""
    d, f = 4096, 14336
    rng = np.random.default_rng(2)
    wn = (1 + 0.1 * rng.standard_normal(d)).astype(np.float32)
    from tensorlisp_b200.native import Native, quantize_rows
    n = Native(0)
    mats = []
    for rows, cols in ((f, d), (f, d), (d, f)):
        w = (rng.standard_normal((rows, cols)) * 0.02).astype(np.float32)
        mats.append(quantize_rows(n, Q4_K, w))   # bit-exact with the oracle (tests/test_gpu_quantize.py)
    n.close()
    x = rng.standard_normal((T, d)).astype(np.float32)
    g = G.Graph()
    tn = g.weight(G.F32, [d], "norm")
    tg = g.weight(G.Q4_K, [d, f], "gate")
    tu = g.weight(G.Q4_K, [d, f], "up")
    td = g.weight(G.Q4_K, [f, d], "down")
    tx = g.input(G.F32, [d, T], "x")
    y = g.output(swiglu_ffn(g, tx, tn, tg, tu, td, 1e-5))
    act = g.output([t for t in g.nodes if g.tensors[t].name == "ffn_act"][0])
    m = Model(g, [wn] + mats)
    got, got_act = m.run(x)
    h = oracle.rms_norm(x, 1e-5, wn)
    a = oracle.mul_mat(Q4_K, mats[0], d, h)
    b = oracle.mul_mat(Q4_K, mats[1], d, h)
    close(got_act, oracle.silu_mul(a, b), 1e-3)
    # the down projection re-quantizes its input: feed the oracle the GPU's own activations
    close(got, oracle.mul_mat(Q4_K, mats[2], f, got_act.reshape(T, f)), 1e-3)
    m.close()


def test_ffn_block_config2_prefill_512(oracle):
    """The same block at 512 tokens (prefill-sized: the tensor-core mul_mat runs 64 columns per launch).
    The CPU check covers a sample of rows of every projection, over all 512 tokens."""
    d, f, T = 4096, 14336, 512
    rng = np.random.default_rng(4)
    wn = (1 + 0.1 * rng.standard_normal(d)).astype(np.float32)
    from tensorlisp_b200.native import Native, quantize_rows
    n = Native(0)
    mats = []
    for rows, cols in ((f, d), (f, d), (d, f)):
        w = (rng.standard_normal((rows, cols)) * 0.02).astype(np.float32)
        mats.append(quantize_rows(n, Q4_K, w))
    n.close()
    x = rng.standard_normal((T, d)).astype(np.float32)
    g = G.Graph()
    tn = g.weight(G.F32, [d], "norm")
    tg = g.weight(G.Q4_K, [d, f], "gate")
    tu = g.weight(G.Q4_K, [d, f], "up")
    td = g.weight(G.Q4_K, [f, d], "down")
    tx = g.input(G.F32, [d, T], "x")
    y = g.output(swiglu_ffn(g, tx, tn, tg, tu, td, 1e-5))
    act = g.output([t for t in g.nodes if g.tensors[t].name == "ffn_act"][0])
    m = Model(g, [wn] + mats)
    got, got_act = m.run(x)
    got, got_act = got.reshape(T, d), got_act.reshape(T, f)
    h = oracle.rms_norm(x, 1e-5, wn)
    rows = rng.choice(f, 48, replace=False)
    a = oracle.mul_mat(Q4_K, mats[0][rows], d, h)
    b = oracle.mul_mat(Q4_K, mats[1][rows], d, h)
    close(got_act[:, rows], oracle.silu_mul(a, b), 1e-3)
    rows = rng.choice(d, 48, replace=False)
    close(got[:, rows], oracle.mul_mat(Q4_K, mats[2][rows], f, got_act), 1e-3)
    m.close()


def test_decode_step(oracle):
    cfg = DecoderConfig(n_layers=2, d_model=512, n_heads=4, n_kv_heads=2, head_dim=128, d_ffn=1024, vocab=1024)
    _decode_step_case(oracle, cfg, np.array([0, 17, 40], np.int32), 64, 4)


def test_decode_step_full_width(oracle):
    """Two layers at the benchmark's own width (d_model 4096, 32 / 8 heads of 128, FFN 14336: the real tile shapes,
    K splits and grouped launches of the 8B-shape step), 8 sequences, a small vocabulary."""
    cfg = DecoderConfig(n_layers=2, d_model=4096, n_heads=32, n_kv_heads=8, head_dim=128, d_ffn=14336, vocab=2048)
    _decode_step_case(oracle, cfg, np.array([0, 5, 31, 100, 255, 16, 77, 200], np.int32), 256, 2)


def _decode_step_case(oracle, cfg, ctx_before, max_ctx, noise_seeds):
    B, bs = len(ctx_before), cfg.block_size
    rng = np.random.default_rng(5)
    pos = ctx_before.copy()                               # tokens already cached per sequence
    lens = ctx_before + 1
    ids = rng.integers(0, cfg.vocab, B).astype(np.int32)
    max_blocks = max_ctx // bs
    pool_blocks = B * max_blocks
    dg = decoder_step(cfg, B, max_ctx, pool_blocks, taps=True)
    weights = make_decoder_weights(oracle, dg.weights, seed=9)
    W = {s.name: (s, w) for s, w in zip(dg.weights, weights)}
    tables = rng.permutation(pool_blocks).astype(np.int32).reshape(B, max_blocks)
    slots = np.array([tables[b, pos[b] // bs] * bs + pos[b] % bs for b in range(B)], np.int64)

    taps = dg.extras["taps"]
    outputs = [("logits", dg.logits), ("token", dg.token)] + list(taps.items())
    m = Model(dg.graph, weights, dg.state_bytes, outputs)
    kvh, hd, heads = cfg.n_kv_heads, cfg.head_dim, cfg.n_heads
    ks = [[np.zeros((lens[b], kvh, hd), np.float16) for b in range(B)] for _ in range(cfg.n_layers)]
    vs = [[np.zeros((lens[b], kvh, hd), np.float16) for b in range(B)] for _ in range(cfg.n_layers)]
    for l in range(cfg.n_layers):
        kp = np.zeros((pool_blocks, kvh, bs, hd), np.float16)
        vp = np.zeros((pool_blocks, kvh, bs, hd), np.float16)
        for b in range(B):
            ks[l][b][:ctx_before[b]] = rng.standard_normal((ctx_before[b], kvh, hd)).astype(np.float16)
            vs[l][b][:ctx_before[b]] = rng.standard_normal((ctx_before[b], kvh, hd)).astype(np.float16)
            for t in range(ctx_before[b]):
                kp[tables[b, t // bs], :, t % bs] = ks[l][b][t]
                vp[tables[b, t // bs], :, t % bs] = vs[l][b][t]
        m.native.state.write(m.native.state_offsets[2 * l], kp)
        m.native.state.write(m.native.state_offsets[2 * l + 1], vp)
    res = m.run(ids, pos, tables, lens, slots.view(np.int32))
    out = {name: r for (name, _), r in zip(outputs, res)}

    def lin(name, x):
        s, w = W[name]
        return oracle.mul_mat(s.ty, w, s.ne[0], np.ascontiguousarray(x, np.float32).reshape(B, s.ne[0]))

    # ---- teacher-forced parity, op by op, on the GPU's own intermediates
    s, w = W["token_embd"]
    assert np.array_equal(out["embd"], oracle.get_rows(s.ty, w, cfg.d_model, ids))
    x = out["embd"]
    for l in range(cfg.n_layers):
        p = "blk.%d." % l
        close(out[p + "attn_in"], oracle.rms_norm(x, cfg.eps, W[p + "attn_norm"][1]), 1e-5)
        h = out[p + "attn_in"]
        for nm, wn in (("q", "wq"), ("k", "wk"), ("v", "wv")):
            close(out[p + nm], lin(p + wn, h), 1e-3)
        close(out[p + "q_rope"], oracle.rope(out[p + "q"].reshape(B, heads, hd), pos, hd, 2, cfg.rope_theta), 1e-5)
        close(out[p + "k_rope"], oracle.rope(out[p + "k"].reshape(B, kvh, hd), pos, hd, 2, cfg.rope_theta), 1e-5)
        kl, vl = copy.deepcopy(ks[l]), copy.deepcopy(vs[l])
        for b in range(B):
            kl[b][pos[b]] = out[p + "k_rope"].reshape(B, kvh, hd)[b].astype(np.float16)
            vl[b][pos[b]] = out[p + "v"].reshape(B, kvh, hd)[b].astype(np.float16)
        _, a32 = oracle.attention_decode(out[p + "q_rope"].reshape(B, heads, hd).astype(np.float16), kl, vl, kvh,
                                         1.0 / np.sqrt(hd))
        a_gpu = out[p + "attn"].astype(np.float32).reshape(B, heads, hd)
        err = np.abs(a_gpu - a32).max()
        assert err <= 1e-3 * np.abs(a32).max() + 2 ** -11 * np.abs(a32).max()   # bar + half an ulp of the f16 output
        close(out[p + "attn_out"], lin(p + "wo", a_gpu.reshape(B, heads * hd)), 1e-3)
        close(out[p + "res1"], x + out[p + "attn_out"], 1e-6)
        x = out[p + "res1"]
        close(out[p + "ffn_in"], oracle.rms_norm(x, cfg.eps, W[p + "ffn_norm"][1]), 1e-5)
        close(out[p + "ffn_gate_out"], lin(p + "ffn_gate", out[p + "ffn_in"]), 1e-3)
        close(out[p + "ffn_up_out"], lin(p + "ffn_up", out[p + "ffn_in"]), 1e-3)
        close(out[p + "ffn_act"], oracle.silu_mul(out[p + "ffn_gate_out"], out[p + "ffn_up_out"]), 1e-5)
        close(out[p + "ffn_down_out"], lin(p + "ffn_down", out[p + "ffn_act"]), 1e-3)
        close(out[p + "res2"], x + out[p + "ffn_down_out"], 1e-6)
        x = out[p + "res2"]
    close(out["final_norm"], oracle.rms_norm(x, cfg.eps, W["output_norm"][1]), 1e-5)
    close(out["logits"], lin("output", out["final_norm"]), 1e-3)
    assert np.array_equal(out["token"].astype(np.int64), out["logits"].argmax(axis=1))

    # ---- end to end from the token ids
    want = oracle_decoder_step(oracle, cfg, dg.weights, weights, ids, pos, copy.deepcopy(ks), copy.deepcopy(vs))
    envelope = 0.0
    for seed in range(noise_seeds):
        noisy = oracle_decoder_step(NoisyOracle(oracle, 1e-6, seed), cfg, dg.weights, weights, ids, pos,
                                    copy.deepcopy(ks), copy.deepcopy(vs))
        envelope = max(envelope, float(np.abs(noisy - want).max()))
    err = float(np.abs(out["logits"] - want).max())
    top2 = np.sort(want, axis=1)[:, -2:]
    decided = (top2[:, 1] - top2[:, 0]) > 2 * max(err, envelope)
    same_top1 = out["logits"].argmax(axis=1) == want.argmax(axis=1)
    plain_bar = err <= 1e-2 and bool(same_top1.all())
    print("decode step d_model %d: end-to-end logits error %.3e (the oracle's own 1e-6-noise envelope %.3e), top-1 equal in %d of %d rows, "
          "%d rows undecided at that noise; the plain bar (1e-2 abs, identical top-1) %s"
          % (cfg.d_model, err, envelope, int(same_top1.sum()), B, int((~decided).sum()), "holds" if plain_bar else "does not hold"))
    assert err <= max(1e-2, 1.5 * envelope), (err, envelope)
    assert np.array_equal(out["logits"].argmax(axis=1)[decided], want.argmax(axis=1)[decided])
    m.close()



@pytest.mark.parametrize("ty", [Q4_K, Q8_0])
def test_a_deep_decoder_stays_at_f32_rounding_from_the_oracle(oracle, ty):
    """32 layers for one sequence. The products are the oracle's integers, so the logits differ by the order of f32 additions only (1e-7),
    unless that flips a code of some activation on the way: then by up to a few 1e-3, as the oracle's own logits do under 1e-7 noise on its
    products. Most draws have no such flip; less precision anywhere would show in all of them."""
    L, ctx = 32, 40
    cfg = DecoderConfig(n_layers=L, d_model=512, n_heads=4, n_kv_heads=2, head_dim=128, d_ffn=1024, vocab=1000, wtype=ty)
    dg = decoder_step(cfg, 1, 64, 4)
    ids, pos = np.array([7], np.int32), np.array([ctx], np.int32)
    far = []
    for seed in range(5):
        rng = np.random.default_rng(seed)
        ws = []
        for s in dg.weights:
            if len(s.ne) == 1:
                ws.append((1 + 0.1 * rng.standard_normal(s.ne[0])).astype(np.float32))
                continue
            # a residual stream that the layers change little, as a trained decoder's
            std = 3.0 if s.name in ("token_embd", "output") else (0.02 / np.sqrt(2 * L) if s.name.endswith(("wo", "ffn_down")) else 0.02)
            ws.append(oracle.quantize(s.ty, (rng.standard_normal((s.ne[1], s.ne[0])) * std).astype(np.float32)))
        ks, vs = ([[rng.standard_normal((ctx + 1, 2, 128)).astype(np.float16)] for _ in range(L)] for _ in range(2))
        m = Model(dg.graph, ws, dg.state_bytes, [("logits", dg.logits)])
        for off, kv in zip(m.native.state_offsets, [x[0] for pair in zip(ks, vs) for x in pair]):
            pool = np.zeros((4, 2, 16, 128), np.float16)
            for i in range(ctx):
                pool[i // 16, :, i % 16] = kv[i]
            m.native.state.write(off, pool)
        (got,) = m.run(ids, pos, np.arange(4, dtype=np.int32).reshape(1, 4), pos + 1, pos.astype(np.int64).view(np.int32))
        m.close()
        want = oracle_decoder_step(oracle, cfg, dg.weights, ws, ids, pos, ks, vs)
        far.append(float(np.linalg.norm(got.reshape(want.shape) - want) / np.linalg.norm(want)))
    print("deep decoder, relative distances from the oracle:", " ".join("%.1e" % f for f in far))
    assert sorted(far)[2] <= 1e-6 and max(far) <= 1e-2, far


def test_attention_quantizes_its_own_output(oracle):
    """Without a context split the paged-attention kernel also quantizes its f16 output rows to Q8_K for the output
    projection (the ROW_QUANT node behind it is folded in: one launch less per layer). TL_NATIVE_NOFUSE=ATTN_QUANT keeps
    the separate launch; both programs must give the same bits."""
    import os
    cfg = DecoderConfig(n_layers=2, d_model=4096, n_heads=32, n_kv_heads=8, head_dim=128, d_ffn=14336, vocab=2048)
    B, max_ctx, bs = 32, 64, cfg.block_size
    rng = np.random.default_rng(21)
    max_blocks = max_ctx // bs
    pool_blocks = B * max_blocks
    ids = rng.integers(0, cfg.vocab, B).astype(np.int32)
    pos = rng.integers(0, max_ctx - 1, B).astype(np.int32)
    lens = pos + 1
    tables = rng.permutation(pool_blocks).astype(np.int32).reshape(B, max_blocks)
    slots = np.array([tables[b, pos[b] // bs] * bs + pos[b] % bs for b in range(B)], np.int64)
    dg = decoder_step(cfg, B, max_ctx, pool_blocks)
    weights = make_decoder_weights(oracle, dg.weights, seed=3)
    pools = [(rng.standard_normal((pool_blocks, cfg.n_kv_heads, bs, cfg.head_dim)) * 0.5).astype(np.float16) for _ in range(2 * cfg.n_layers)]
    got, counts = [], []
    for separate in (False, True):
        if separate:
            os.environ["TL_NATIVE_NOFUSE"] = "ATTN_QUANT"
        try:
            m = Model(dg.graph, weights, dg.state_bytes, [("logits", dg.logits)])
        finally:
            os.environ.pop("TL_NATIVE_NOFUSE", None)
        for i, pl in enumerate(pools):
            m.native.state.write(m.native.state_offsets[i], pl)
        (logits,) = m.run(ids, pos, tables, lens, slots.view(np.int32))
        got.append(logits.copy())
        counts.append(m.program.kernel_count())
        m.close()
    assert np.array_equal(got[0], got[1])
    assert np.isfinite(got[0]).all() and np.abs(got[0]).max() > 0
    assert counts[1] - counts[0] == cfg.n_layers, counts
