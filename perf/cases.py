"""What is timed: the work a program that links this framework gives it, over the sizes it is given in use.

Every case goes through the public Python entry points (``Native``, ``NativeProgram``, ``EntryCache``,
``quantize_rows``) the way the model runner of the reference drives its native executor: weights, state and the
compiled program are kept from call to call, the inputs of a call are host arrays, and its results are read back
to the host. Families:

  matmul     one quantized or plain matrix times a few activation columns
  ffn        a gated feed-forward block
  attention  paged-attention decode over a ragged batch
  decode     one step of a whole decoder over a paged KV pool, sampled on the host or greedy
  prompt     the prompt pass of a whole decoder
  quantize   f32 rows to GGUF blocks, host to host

Weights are normal and go through the library's own quantizers, keys and values are N(0, 1) pages in a random
order, token ids are uniform over the vocabulary. Decoders use tied embeddings and scale the projections that write
the residual stream with the depth, as initialisations for training do, beside embeddings of a larger scale: the best
token then has a margin, as it has in a trained model, and a code of an 8-bit activation that rounds the other way
stays a small difference through all the layers.
"""
import ctypes as C
import math

import numpy as np
import torch

from tensorlisp_b200 import graph as G
from tensorlisp_b200._lib import check
from tensorlisp_b200.native import EntryCache, Native, NativeProgram, StateBlock, quantize_rows
from tensorlisp_b200.programs import DecoderConfig, decoder_step, decoder_weights, prefill_step, swiglu_ffn

TYPES = {"f16": G.F16, "bf16": G.BF16, "q4_0": G.Q4_0, "q8_0": G.Q8_0, "q4_K": G.Q4_K, "q5_K": G.Q5_K, "q6_K": G.Q6_K}


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest call: a single-op program, one activation vector (benchmark configuration 1)
        dict(name="matmul_q8_0_1", kind="matmul", type="q8_0", k=4096, m=4096, n=1),
        # the same matrix in the smallest block type for a batch of 16
        dict(name="matmul_q4_0_16", kind="matmul", type="q4_0", k=4096, m=4096, n=16),
        # a layer matrix that was left in half precision, a small decode batch
        dict(name="matmul_f16_8", kind="matmul", type="f16", k=4096, m=14336, n=8),
        # mixed-type files keep their most sensitive matrices, the output projection among them, in Q6_K
        dict(name="matmul_q6_K_1", kind="matmul", type="q6_K", k=4096, m=32000, n=1),
        # the feed-forward block for one token and for a prompt chunk (benchmark configuration 2)
        dict(name="ffn_q4_K_1", kind="ffn", type="q4_K", d=4096, ffn=14336, n=1),
        dict(name="ffn_q4_K_512", kind="ffn", type="q4_K", d=4096, ffn=14336, n=512),
        # attention of a serving batch with very different context lengths (benchmark configuration 3)
        dict(name="attention_64_ragged", kind="attention", seqs=64, ctx=8192, heads=32, kv_heads=8, hs=128),
        # one user's chat: a step of the whole decoder at batch 1, the logits sampled on the host
        dict(name="decode_q4_K_1", kind="decode", type="q4_K", layers=32, d=4096, heads=32, kv_heads=8, hs=128, ffn=14336, vocab=128256,
             batch=1, ctx=1024, ragged=False, greedy=False),
        # the serving step: batch 32 at context 2048, greedy (benchmark configuration 4)
        dict(name="decode_q4_K_32", kind="decode", type="q4_K", layers=32, d=4096, heads=32, kv_heads=8, hs=128, ffn=14336, vocab=128256,
             batch=32, ctx=2048, ragged=False, greedy=True),
        # a chat turn's prompt of a length that fits no tile
        dict(name="prompt_q4_K_1x333", kind="prompt", type="q4_K", layers=32, d=4096, heads=32, kv_heads=8, hs=128, ffn=14336, vocab=128256,
             seqs=1, tokens=333),
        # the batched prompt pass (benchmark configuration 5)
        dict(name="prompt_q8_0_8x2048", kind="prompt", type="q8_0", layers=32, d=4096, heads=32, kv_heads=8, hs=128, ffn=14336, vocab=128256,
             seqs=8, tokens=2048),
        # converting a checkpoint: one layer matrix
        dict(name="quantize_q4_K", kind="quantize", type="q4_K", rows=14336, n=4096),
    ]


def _log(rng, lo, hi, step=1):
    """A multiple of `step` in [lo, hi], uniform in the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


# widths that the repository's tests and benchmark use, and two between them
WIDTHS = [dict(d=512, heads=4, kv_heads=2, hs=128, ffn=1024), dict(d=1024, heads=16, kv_heads=4, hs=64, ffn=2816),
          dict(d=2048, heads=16, kv_heads=4, hs=128, ffn=5632), dict(d=4096, heads=32, kv_heads=8, hs=128, ffn=14336)]


def draw(rng):
    kind = rng.choice(["matmul", "matmul", "matmul", "ffn", "ffn", "attention", "decode", "decode", "prompt", "quantize"])
    if kind == "matmul":
        # row lengths are whole super-blocks of 256, row counts are anything
        return dict(kind=kind, type=rng.choice(["q8_0", "q4_0", "q4_K", "q6_K", "f16", "bf16"]), k=_log(rng, 512, 14336, 256), m=_log(rng, 500, 32000),
                    n=_log(rng, 1, 64))
    if kind == "ffn":
        d = _log(rng, 512, 4096, 256)
        return dict(kind=kind, type=rng.choice(["q4_K", "q8_0"]), d=d, ffn=_log(rng, 2 * d, 3.5 * d, 256), n=_log(rng, 1, 512))
    if kind == "attention":
        h = rng.choice([dict(heads=32, kv_heads=8, hs=128), dict(heads=16, kv_heads=4, hs=64), dict(heads=8, kv_heads=8, hs=128), dict(heads=16, kv_heads=2, hs=128)])
        return dict(kind=kind, seqs=_log(rng, 1, 64), ctx=_log(rng, 100, 8192), **h)
    if kind == "decode":
        w = rng.choice(WIDTHS)
        return dict(kind=kind, type=rng.choice(["q4_K", "q4_K", "q8_0"]), layers=_log(rng, 2, 32), vocab=_log(rng, 1000, 128256, 8), batch=_log(rng, 1, 32),
                    ctx=_log(rng, 64, 2048), ragged=rng.random() < 0.5, greedy=rng.random() < 0.5, **w)
    if kind == "prompt":
        w = rng.choice(WIDTHS)
        seqs = _log(rng, 1, 8)
        return dict(kind=kind, type=rng.choice(["q4_K", "q8_0"]), layers=_log(rng, 2, 32), vocab=_log(rng, 1000, 128256, 8), seqs=seqs, tokens=_log(rng, 16, 2048), **w)
    n = _log(rng, 256, 14336, 256)
    return dict(kind=kind, type=rng.choice(["q4_K", "q8_0", "q4_0", "q6_K", "q5_K", "f16"]), rows=_log(rng, 32, min(14336, 14336 * 4096 // n)), n=n)


# ------------------------------------------------------------------------------------------------ helpers
class _Device:
    """Device memory of the library as an array that torch can wrap; the tensor keeps `owner` (and so the memory) alive."""

    def __init__(self, owner, ptr, shape, typestr, strides=None):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=tuple(shape), typestr=typestr, data=(ptr, False), version=3, strides=strides)


def _device(owner, ptr, shape, typestr, strides=None):
    return torch.as_tensor(_Device(owner, ptr, shape, typestr, strides), device="cuda")


def _generator(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 1000003 + salt)
    return g


def _matrix(native, ptr, ty, m, k, std, gen):
    """A normal [m, k] matrix written to device memory at `ptr` in ggml type `ty`."""
    row = G.row_size(ty, k)
    for r in range(0, m, 32768):
        w = torch.randn((min(m - r, 32768), k), generator=gen, device="cuda") * std
        if ty in (G.F16, G.BF16):
            _device(native.weights, ptr + r * row, w.shape, "<i2").copy_(w.to(torch.float16 if ty == G.F16 else torch.bfloat16).view(torch.int16))
            continue
        torch.cuda.current_stream().synchronize()
        check(native.L.tlb_quantize_rows_device(native.dev, ty, C.c_void_p(w.data_ptr()), w.shape[0], k, C.c_void_p(ptr + r * row)))
        native.sync()


def _weights(native, specs, seed, std):
    """The weight buffer: every tensor at a 256-byte aligned offset, norms N(1, 0.1), matrices N(0, std(name))."""
    total = 0
    for s in specs:
        native.weight_loc.append((0, total))
        total += G.align256(s[2])
    h = C.c_void_p()
    check(native.L.tlb_weights_create(native.dev, total, C.byref(h)))
    native.weights = StateBlock(h)
    for i, ((name, ty, nbytes, ne), (_, off)) in enumerate(zip(specs, native.weight_loc)):
        ptr = native.weights.device_ptr + off
        gen = _generator(seed, 0 if name == "output" else i)      # the output projection is the embedding matrix
        if len(ne) == 1:
            _device(native.weights, ptr, ne, "<f4").copy_(1 + 0.1 * torch.randn(ne[0], generator=gen, device="cuda"))
        else:
            _matrix(native, ptr, ty, ne[1], ne[0], std(name), gen)
    torch.cuda.current_stream().synchronize()


def _spec(name, ty, ne):
    return (name, ty, G.row_size(ty, ne[0]) * (ne[1] if len(ne) > 1 else 1), ne)


def _decoder(case, seed, native, dg):
    L = case["layers"]

    def std(name):
        if name in ("token_embd", "output"):
            return 3.0
        return 0.02 / math.sqrt(2 * L) if name.endswith(("wo", "ffn_down")) else 0.02

    _weights(native, [_spec(s.name, s.ty, s.ne) for s in dg.weights], seed, std)
    native.alloc_states(dg.state_bytes)


def _config(case):
    return DecoderConfig(n_layers=case["layers"], d_model=case["d"], n_heads=case["heads"], n_kv_heads=case["kv_heads"], head_dim=case["hs"],
                         d_ffn=case["ffn"], vocab=case["vocab"], wtype=TYPES[case["type"]])


def _lengths(rng, seqs, ctx, ragged):
    """Context lengths; the ragged ones are spread evenly over [ctx / 64, ctx] in a random order, so that their sum is the case's own."""
    if not ragged:
        return np.full(seqs, ctx, np.int32)
    return rng.permutation(_spread(seqs, ctx)).astype(np.int32)


def _spread(seqs, ctx):
    return np.rint(np.linspace(ctx, max(1, ctx // 64), seqs)).astype(np.int64)


def _total(seqs, ctx, ragged):
    return int(_spread(seqs, ctx).sum()) if ragged else seqs * ctx


# ------------------------------------------------------------------------------------------------ prepare
def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def _prepare_matmul(case, seed):
    ty, k, m, n = TYPES[case["type"]], case["k"], case["m"], case["n"]
    native = Native(0)
    _weights(native, [_spec("W", ty, [k, m])], seed, lambda name: 0.02)

    def build(name, shapes):
        g = G.Graph()
        w = g.weight(ty, [k, m], "W")
        g.output(g.mul_mat(w, g.input(G.F32, [k, n], "x"), "y"))
        return g

    x = torch.randn((n, k), generator=_generator(seed, 77), device="cuda").cpu().numpy()
    return dict(kind="entry", cache=EntryCache(native, build), inputs=[x], native=native)


def _prepare_ffn(case, seed):
    ty, d, f, n = TYPES[case["type"]], case["d"], case["ffn"], case["n"]
    native = Native(0)
    _weights(native, [_spec("norm", G.F32, [d]), _spec("gate", ty, [d, f]), _spec("up", ty, [d, f]), _spec("down", ty, [f, d])], seed, lambda name: 0.02)

    def build(name, shapes):
        g = G.Graph()
        w = [g.weight(G.F32, [d], "norm"), g.weight(ty, [d, f], "gate"), g.weight(ty, [d, f], "up"), g.weight(ty, [f, d], "down")]
        g.output(swiglu_ffn(g, g.input(G.F32, [d, n], "x"), *w, 1e-5))
        return g

    x = torch.randn((n, d), generator=_generator(seed, 77), device="cuda").cpu().numpy()
    return dict(kind="entry", cache=EntryCache(native, build), inputs=[x], native=native)


def _prepare_attention(case, seed):
    seqs, ctx, heads, kvh, hs, bs = case["seqs"], case["ctx"], case["heads"], case["kv_heads"], case["hs"], 16
    rng = np.random.default_rng(seed)
    lens = _lengths(rng, seqs, ctx, True)
    max_blocks = (ctx + bs - 1) // bs
    need = (lens.astype(np.int64) + bs - 1) // bs
    pool_blocks = int(need.sum())
    pages = rng.permutation(pool_blocks).astype(np.int32)
    tables = np.zeros((seqs, max_blocks), np.int32)
    at = 0
    for s in range(seqs):
        tables[s, :need[s]] = pages[at:at + need[s]]
        at += need[s]
    g = G.Graph()
    pool = pool_blocks * kvh * bs * hs
    kc, vc = g.state(G.F16, [pool], "k_pool"), g.state(G.F16, [pool], "v_pool")
    q = g.input(G.F32, [hs, heads, seqs], "q")
    tt, tl = g.input(G.I32, [max_blocks, seqs], "tables"), g.input(G.I32, [seqs], "lens")
    out = g.output(g.cast(g.paged_attention(g.cast(q, G.F16), kc, vc, tt, tl, bs, ctx, 1.0 / math.sqrt(hs), kvh), G.F32, "attn"))
    native = Native.load([])
    native.alloc_states([pool * 2] * 2)
    for i, off in enumerate(native.state_offsets):
        _device(native.state, native.state.device_ptr + off, (pool,), "<f2").normal_(generator=_generator(seed, i))
    torch.cuda.current_stream().synchronize()
    prog = NativeProgram.compile(native, g)
    inputs = [rng.standard_normal((seqs, heads, hs)).astype(np.float32), tables, lens]
    return dict(kind="attention", prog=prog, native=native, inputs=inputs, out=out)


def _prepare_decode(case, seed):
    cfg, B, ctx = _config(case), case["batch"], case["ctx"]
    bs = cfg.block_size
    max_blocks = (ctx + bs - 1) // bs
    pool_blocks = B * max_blocks
    dg = decoder_step(cfg, B, ctx, pool_blocks, with_argmax=case["greedy"])
    native = Native(0)
    _decoder(case, seed, native, dg)
    base = native.state.device_ptr
    pool = dg.state_bytes[0] // 2
    for i, off in enumerate(native.state_offsets):
        _device(native.state, base + off, (pool,), "<f2").normal_(generator=_generator(seed, 500 + i))
    torch.cuda.current_stream().synchronize()
    prog = NativeProgram.compile(native, dg.graph)
    rng = np.random.default_rng(seed)
    lens = _lengths(rng, B, ctx, case["ragged"])
    pos = lens - 1
    # a random order of the pages, except that the page a sequence writes this step is page b of the pools
    tables = np.zeros((B, max_blocks), np.int32)
    rest = iter(rng.permutation(np.arange(B, pool_blocks)).astype(np.int32))
    for b in range(B):
        for j in range(max_blocks):
            tables[b, j] = b if j == pos[b] // bs else next(rest)
    slots = tables[np.arange(B), pos // bs].astype(np.int64) * bs + pos % bs
    inputs = [rng.integers(0, cfg.vocab, B).astype(np.int32), pos.astype(np.int32), tables, lens, slots.view(np.int32)]
    # the pages that this step writes to, of every pool
    step = native.state_offsets[1] - native.state_offsets[0] if len(native.state_offsets) > 1 else dg.state_bytes[0]
    page = cfg.n_kv_heads * bs * cfg.head_dim
    written = _device(native.state, base, (len(native.state_offsets), B * page), "<f2", (step, 2))
    ptr, _ = prog.tensor_ptr(dg.logits)
    logits = _device(prog, ptr, (B, cfg.vocab), "<f4")
    return dict(kind="decode", prog=prog, native=native, inputs=inputs, token=dg.token, logits=dg.logits, logits_view=logits, written=written, greedy=case["greedy"])


def _prepare_prompt(case, seed):
    cfg, S, T = _config(case), case["seqs"], case["tokens"]
    bs = cfg.block_size
    dg = prefill_step(cfg, S, T)
    native = Native(0)
    _decoder(case, seed, native, dg)
    prog = NativeProgram.compile(native, dg.graph)
    rng = np.random.default_rng(seed)
    per = (T + bs - 1) // bs
    tables = rng.permutation(S * per).astype(np.int64).reshape(S, per)
    t = np.arange(T)
    slots = (tables[:, t // bs] * bs + t % bs).reshape(-1)
    # positions, mask and row numbers belong to the shape: they are set once
    prog.set_input(dg.inputs["pos"], np.tile(t.astype(np.int32), S))
    prog.set_input(dg.inputs["mask"], np.triu(np.full((T, T), -np.inf, np.float16), 1))
    prog.set_input(dg.inputs["last"], (np.arange(S) * T + T - 1).astype(np.int32))
    step = native.state_offsets[1] - native.state_offsets[0]
    pools = _device(native.state, native.state.device_ptr, (len(native.state_offsets), dg.state_bytes[0] // 2), "<f2", (step, 2))
    return dict(kind="prompt", prog=prog, native=native, ids=rng.integers(0, cfg.vocab, S * T).astype(np.int32), slots=slots.view(np.int32),
                at=dg.inputs, logits=dg.logits, pools=pools)


def _prepare_quantize(case, seed):
    x = torch.randn((case["rows"], case["n"]), generator=_generator(seed, 5), device="cuda") * 0.02
    return dict(kind="quantize", native=Native(0), type=TYPES[case["type"]], x=x.cpu().numpy())


# ------------------------------------------------------------------------------------------------ run
def run(state):
    kind = state["kind"]
    if kind == "entry":
        return {name: y for name, y in state["cache"].run("entry", state["inputs"])}
    if kind == "quantize":
        return {"blocks": quantize_rows(state["native"], state["type"], state["x"])}
    prog = state["prog"]
    if kind == "prompt":
        prog.set_input(state["at"]["ids"], state["ids"])
        prog.set_input(state["at"]["slots"], state["slots"])
        prog.run()
        return {"logits": prog.read(state["logits"]), "cache": state["pools"]}
    for i, a in enumerate(state["inputs"]):
        prog.set_input(i, a)
    prog.run()
    if kind == "attention":
        return {"attention": prog.read(state["out"])}
    if state["greedy"]:
        return {"token": prog.read(state["token"]).astype(np.int64), "logits": state["logits_view"], "cache": state["written"]}
    return {"logits": prog.read(state["logits"]), "cache": state["written"]}


# ------------------------------------------------------------------------------------------------ work, tolerance
def work(case):
    kind = case["kind"]
    if kind == "matmul":
        k, m, n = case["k"], case["m"], case["n"]
        return {"bytes": G.row_size(TYPES[case["type"]], k) * m + 4 * (k + m) * n, "flops": 2 * k * m * n}
    if kind == "ffn":
        d, f, n = case["d"], case["ffn"], case["n"]
        ty = TYPES[case["type"]]
        return {"bytes": 2 * G.row_size(ty, d) * f + G.row_size(ty, f) * d + 4 * d + 8 * d * n, "flops": 6 * d * f * n}
    if kind == "quantize":
        return {"bytes": case["rows"] * (4 * case["n"] + G.row_size(TYPES[case["type"]], case["n"])), "flops": 0}
    heads, kvh, hs = case["heads"], case["kv_heads"], case["hs"]
    if kind == "attention":
        total = _total(case["seqs"], case["ctx"], True)
        return {"bytes": total * kvh * hs * 4 + case["seqs"] * heads * hs * 8, "flops": 4 * total * heads * hs}
    cfg = _config(case)
    mats = [s for s in decoder_weights(cfg) if s.name != "token_embd"]
    nbytes = sum(s.nbytes() for s in mats)
    layer = sum(s.ne[0] * s.ne[1] for s in mats if len(s.ne) == 2 and s.name != "output")
    if kind == "decode":
        B = case["batch"]
        total = _total(B, case["ctx"], case["ragged"])
        return {"bytes": nbytes + cfg.n_layers * total * kvh * hs * 4 + B * G.row_size(cfg.etype, cfg.d_model) + 4 * B * cfg.vocab,
                "flops": 2 * B * (layer + cfg.d_model * cfg.vocab) + 4 * cfg.n_layers * total * heads * hs}
    S, T = case["seqs"], case["tokens"]
    return {"bytes": nbytes + cfg.n_layers * S * T * kvh * hs * 4 + S * T * G.row_size(cfg.etype, cfg.d_model) + 4 * S * cfg.vocab,
            "flops": 2 * S * (T * layer + cfg.d_model * cfg.vocab) + 2 * cfg.n_layers * S * T * (T + 1) * heads * hs}


def tolerance(case):
    kind = case["kind"]
    if kind == "quantize":
        return "exact"
    if kind == "matmul":
        # the integer sums of a block are exact, the rest is f32 (f16, bf16 and Q6_K weights meet f32 activations)
        return {"rel": 1e-5}
    if kind == "attention":
        return {"rel": 1e-3}        # f16 queries, pages and result
    if kind == "ffn":
        # the input of the second product is rounded to 8-bit codes again: a last-bit difference moves some of them by a step
        return {"rel": 2e-3 if case["n"] <= 64 else 5e-3}
    # a whole decoder repeats that rounding before every product
    return {"rel": 2e-2}
