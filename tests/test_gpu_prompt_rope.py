"""The rope, casts and cache write of a prompt in one launch against the separate ones: the same bytes in the pools, the same logits.
Head sizes of half a CTA's row and less, an odd number of tokens, tokens without a slot."""
import numpy as np
import pytest

from helpers import Model, make_decoder_weights
from tensorlisp_b200.graph import Q8_0
from tensorlisp_b200.programs import DecoderConfig, prefill_step

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd,heads,kvh,n_seqs,n_tokens", [(64, 8, 4, 1, 33), (128, 4, 2, 3, 37), (128, 8, 8, 2, 16)])
def test_one_launch_or_five(oracle, monkeypatch, hd, heads, kvh, n_seqs, n_tokens):
    cfg = DecoderConfig(n_layers=2, d_model=512, n_heads=heads, n_kv_heads=kvh, head_dim=hd, d_ffn=512, vocab=512, wtype=Q8_0)
    dg = prefill_step(cfg, n_seqs, n_tokens)
    weights = make_decoder_weights(oracle, dg.weights, seed=3)
    rng = np.random.default_rng(hd + n_tokens)
    T, bs = n_seqs * n_tokens, cfg.block_size
    per = (n_tokens + bs - 1) // bs
    tables = rng.permutation(n_seqs * per).astype(np.int64).reshape(n_seqs, per)
    t = np.arange(n_tokens)
    slots = (tables[:, t // bs] * bs + t % bs).reshape(-1)
    slots[1::7] = -1
    ins = (rng.integers(0, cfg.vocab, T).astype(np.int32), np.tile(np.arange(n_tokens, dtype=np.int32), n_seqs),
           np.triu(np.full((n_tokens, n_tokens), -np.inf, np.float16), 1), (np.arange(n_seqs) * n_tokens + n_tokens - 1).astype(np.int32), slots.view(np.int32))
    seen, counts = [], []
    for off in ("", "ROPE_KV_WRITE"):
        monkeypatch.setenv("TL_NATIVE_NOFUSE", off)
        m = Model(dg.graph, weights, dg.state_bytes)
        out = [m.run(*ins)[0].copy()]
        out += [m.native.state.read(o, n) for o, n in zip(m.native.state_offsets, dg.state_bytes)]
        counts.append(m.program.kernel_count())
        seen.append(out)
        m.close()
    assert counts[0] == counts[1] - 4 * cfg.n_layers
    for a, b in zip(*seen):
        assert np.asarray(a).tobytes() == np.asarray(b).tobytes()
