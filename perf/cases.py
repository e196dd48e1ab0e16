"""What a user of this package has it do, as timed cases: dequantizing GEMVs, decode steps, prompts, verify windows, MoE blocks.

A case is a plain dict.  `prepare` makes its inputs from a seed, `run` is one pass through the public entry points (`QMat`, `Model`,
`State`), `work` the bytes and operations a pass cannot do without, `tolerance` how far another correct implementation at the same
precision may be off.  Kinds and ranges:

  gemv    y = W x for one quantized matrix: formats IQ3_S, IQ2_XS, Q4_K, Q8_0; any number of rows from an expert's to the
          vocabulary's; 1 to 128 tokens; on device pointers, or through the host-buffer form (host = True)
  decode  greedy tokens of 1 to 32 sequences over a 4-bit KV cache of up to 32768 positions, on the device
  step    one token in, its logits out on the host: the call of a host-side sampler
  prompt  a prompt of up to 4096 tokens into a fresh state (prefix = 0) or behind a restored snapshot (prefix = its length)
  verify  a window of 2 to 8 drafted tokens and the rollback to those that were kept
  moe     one MoE block on 1 to 128 tokens: router, top-10 of 512 experts, SwiGLU, shared expert

The model is one period (three Gated DeltaNet layers, one attention layer, a MoE block behind each) of the benchmark's decoder in its
full width, with embedding and lm-head, so that a pass is short and three models fit one GPU; weights are random-init, in IQ3_S or Q4_K.
"""
import math

import numpy as np
import torch

import pyre_b200 as pb
from pyre_b200 import synth

BLOCK = {"IQ3_S": (256, 110), "IQ2_XS": (256, 74), "Q4_K": (256, 144), "Q8_0": (32, 34)}   # elements, bytes of a block
D, FF, N_EXP, TOP_K, VOCAB, LAYERS = 2048, 512, 512, 10, 151936, 4
ROOM = 768          # positions a decode or verify state advances before it is set back to its context (inside the f32 window of the cache)

_ctx = None


def _context():
    """The process's context: a program makes one and keeps it."""
    global _ctx
    if _ctx is None:
        _ctx = pb.Ctx(0)
    return _ctx


def listed():
    return [
        # the smallest call: the down projection of one expert for one token; launch and host overhead decide
        dict(name="gemv_expert_down", kind="gemv", type="Q8_0", rows=2048, cols=512, t=1, host=False),
        # the host-buffer form that the engine's callers have, a projection of a window of four tokens
        dict(name="gemv_projection_host", kind="gemv", type="Q4_K", rows=4096, cols=2048, t=4, host=True),
        # the lm-head of one decode step, the largest single matrix
        dict(name="gemv_lm_head", kind="gemv", type="IQ3_S", rows=151936, cols=2048, t=1, host=False),
        # the lm-head of a decode batch
        dict(name="gemv_lm_head_batch16", kind="gemv", type="IQ2_XS", rows=151936, cols=2048, t=16, host=False),
        # an odd number of tokens against an odd number of rows: the fused input projections of a ragged prompt piece
        dict(name="gemv_ragged_prompt", kind="gemv", type="IQ3_S", rows=12351, cols=2048, t=77, host=False),
        # one user, long context: the headline decode loop
        dict(name="decode_bs1_ctx32768", kind="decode", type="IQ3_S", batch=1, ctx=32768, n=16),
        # many users, long contexts
        dict(name="decode_bs32_ctx32768", kind="decode", type="IQ3_S", batch=32, ctx=32768, n=4),
        # interactive decoding with the sampler on the host, short context, the other common format
        dict(name="step_bs1_ctx500", kind="step", type="Q4_K", batch=1, ctx=500),
        # a long prompt from nothing
        dict(name="prompt_4096", kind="prompt", type="IQ3_S", prefix=0, t=4096),
        # the next turn of a conversation: cached prefix, then an odd number of new tokens
        dict(name="prompt_333_after_2048", kind="prompt", type="IQ3_S", prefix=2048, t=333),
        # speculative decoding: six drafted tokens, four kept
        dict(name="verify_6_keep_4_ctx8192", kind="verify", type="IQ3_S", t=6, keep=4, ctx=8192),
        # the MoE block of the layer benchmark
        dict(name="moe_128_tokens", kind="moe", type="IQ3_S", t=128),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["gemv", "gemv", "gemv", "decode", "decode", "step", "prompt", "prompt", "verify", "moe"])
    wtype = rng.choice(["IQ3_S", "IQ3_S", "IQ3_S", "Q4_K"])
    if kind == "gemv":
        return dict(kind=kind, type=rng.choice(sorted(BLOCK)), rows=_log_int(rng, 512, 151936), cols=rng.choice([512, 1024, 2048, 4096]),
                    t=_log_int(rng, 1, 128), host=rng.random() < 0.25)
    if kind == "decode":
        return dict(kind=kind, type=wtype, batch=_log_int(rng, 1, 32), ctx=_log_int(rng, 64, 32768), n=rng.randint(4, 16))
    if kind == "step":
        return dict(kind=kind, type=wtype, batch=_log_int(rng, 1, 8), ctx=_log_int(rng, 64, 32768))
    if kind == "prompt":
        return dict(kind=kind, type=wtype, prefix=256 * rng.choice([0, 0, rng.randint(1, 16)]), t=_log_int(rng, 3, 3840))
    if kind == "verify":
        t = rng.randint(2, 8)
        return dict(kind=kind, type=wtype, t=t, keep=rng.randint(1, t), ctx=_log_int(rng, 64, 32768))
    return dict(kind=kind, type=wtype, t=_log_int(rng, 1, 128))


class _Held:
    """A model with its state, released with the last reference."""

    def __init__(self, case, seed, max_ctx, batch):
        ctx = _context()
        cfg = pb.make_cfg(n_layers=LAYERS, d=D, n_exp=N_EXP, top_k=TOP_K, ff_exp=FF, ff_sh=FF, vocab=VOCAB, max_ctx=max_ctx, kv_bits=4, kv_recent=1024)
        self.model = synth.build_model(ctx, cfg, synth.model_spec(cfg, seed, getattr(pb, case["type"])), seed)
        self.st = self.model.new_state(batch)

    def __del__(self):
        if hasattr(self, "st"):
            self.st.destroy()
        if hasattr(self, "model"):
            self.model.destroy()


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind, ctx = case["kind"], _context()
    s = dict(case=case)
    if kind == "gemv":
        s["w"] = _Matrix(ctx, case, seed)
        if case["host"]:
            s["x"] = rng.standard_normal((case["t"], case["cols"])).astype(np.float32)
        else:
            g = torch.Generator(device="cuda").manual_seed(seed)
            s["x"] = torch.randn(case["t"], case["cols"], device="cuda", generator=g)
            s["y"] = torch.empty(case["t"], case["rows"], device="cuda")
        torch.cuda.synchronize()
        ctx.sync()
        return s
    batch = case["t"] if kind == "moe" else case.get("batch", 1)
    filled = case.get("ctx", case.get("prefix", 0))
    h = s["held"] = _Held(case, seed, filled + (case["t"] if kind == "prompt" else ROOM) + 64, batch)
    if kind == "moe":
        s["x"] = rng.standard_normal((case["t"], D)).astype(np.float32)
    elif kind == "prompt":
        s["ids"] = rng.integers(0, VOCAB, case["t"], dtype=np.uint32)
    else:
        s["ids"] = rng.integers(0, VOCAB, case["t"] if kind == "verify" else batch, dtype=np.uint32)
    if filled:
        h.st.fill_kv_synth(0, filled, seed)
        h.st.set_pos(filled)
    if kind == "prompt" and filled:
        s["blob"] = h.st.snapshot()
    if kind == "step":
        s["out"] = ctx.pinned_empty((batch, VOCAB))
    s["pos"] = filled
    ctx.sync()
    return s


class _Matrix:
    """A matrix on the GPU, released with the last reference."""

    def __init__(self, ctx, case, seed):
        self.m = pb.QMat.synth(ctx, getattr(pb, case["type"]), case["rows"], case["cols"], seed, 1)

    def __del__(self):
        if hasattr(self, "m"):
            self.m.free()


def _advance(s, n):
    """The sequences go on where the last pass left them; near the end of the cache they are set back to their context."""
    c = s["case"]
    if s["pos"] + n > c["ctx"] + ROOM:
        s["held"].st.set_pos(c["ctx"])
        s["pos"] = c["ctx"]


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "gemv":
        if c["host"]:
            return s["w"].m.matmul(s["x"])
        s["w"].m.matmul_dev(s["x"].data_ptr(), c["t"], s["y"].data_ptr())
        return s["y"]
    st = s["held"].st
    if kind == "decode":
        _advance(s, c["n"])
        tok = st.decode_greedy(s["ids"], c["n"])
        s["pos"] += c["n"]
        return tok.astype(np.int64)
    if kind == "step":
        _advance(s, 1)
        s["pos"] += 1
        return st.forward(s["ids"].reshape(-1, 1), out=s["out"])
    if kind == "prompt":
        if c["prefix"]:
            st.restore(s["blob"])
        else:
            st.reset()
        return st.forward(s["ids"])
    if kind == "verify":
        _advance(s, c["t"])
        logits = st.forward_multi(s["ids"])
        st.spec_keep(c["t"], c["keep"])
        s["pos"] += c["keep"]
        return logits
    y, sel = st.moe_forward(0, s["x"])
    return {"y": y, "experts": sel}


def _row_bytes(t, cols):
    e, b = BLOCK[t]
    return cols // e * b


def _distinct(tokens):
    """Expected number of distinct routed experts of `tokens` tokens."""
    return N_EXP * (1.0 - (1.0 - TOP_K / N_EXP) ** tokens)


def _moe_bytes(t, tokens):
    expert = 2 * FF * _row_bytes(t, D) + D * _row_bytes(t, FF)
    return N_EXP * D * 4 + (_distinct(tokens) + 1) * expert


_DENSE = {"lin": (2 * 16 * 128 + 32 * 128 + 32 * 128 + 64, 32 * 128), "attn": (16 * 2 * 256 + 2 * 2 * 256, 16 * 256)}   # input projection rows, output projection columns


def _layer_bytes(t):
    return sum(n * (r * _row_bytes(t, D) + D * _row_bytes(t, o)) for n, (r, o) in ((3, _DENSE["lin"]), (1, _DENSE["attn"])))


def _token_flops():
    dense = sum(n * D * (r + o) for n, (r, o) in ((3, _DENSE["lin"]), (1, _DENSE["attn"])))
    return 2.0 * (dense + LAYERS * ((TOP_K + 1) * 3 * D * FF + N_EXP * D)) + 3 * 8.0 * 32 * 128 * 128


def _kv_bytes(ctx):
    packed = max(0, (ctx - 1024) // 64 * 64)
    return 2 * 2 * (packed * (128 + 32) + (ctx - packed) * 1024)


_STATE = 3 * 2 * (32 * 128 * 128 + 4 * 8192) * 4     # recurrent state of the DeltaNet layers, read and written


def _pass(t, tokens, seqs, kv_positions, head_rows, scored):
    """One pass of the model: `tokens` tokens of `seqs` sequences that read `kv_positions` cached positions each and attend to `scored`
    positions in all, `head_rows` rows of logits."""
    b = _layer_bytes(t) + LAYERS * _moe_bytes(t, tokens) + VOCAB * _row_bytes(t, D) + seqs * (_kv_bytes(kv_positions) + _STATE)
    b += head_rows * VOCAB * 4 + tokens * _row_bytes(t, D)
    return b, tokens * _token_flops() + head_rows * 2.0 * VOCAB * D + scored * 4.0 * 16 * 256


def work(case):
    kind, t = case["kind"], case["type"]
    if kind == "gemv":
        n, r, c = case["t"], case["rows"], case["cols"]
        return {"bytes": r * _row_bytes(t, c) + 4 * n * (r + c), "flops": 2.0 * r * c * n}
    if kind == "moe":
        n = case["t"]
        return {"bytes": _moe_bytes(t, n) + 2 * n * D * 4, "flops": 2.0 * n * ((TOP_K + 1) * 3 * D * FF + N_EXP * D)}
    if kind in ("decode", "step"):
        n = case.get("n", 1)
        b, f = _pass(t, case["batch"], case["batch"], case["ctx"], case["batch"], case["batch"] * case["ctx"])
        return {"bytes": n * b, "flops": n * f}
    n, before = case["t"], case.get("prefix", case.get("ctx", 0))
    b, f = _pass(t, n, 1, before + (n if kind == "prompt" else 0), n if kind == "verify" else 1, n * before + n * n / 2)
    if kind == "verify":
        b += (n - 1) * _STATE // 2     # the rollback checkpoints
    elif before:
        b += _kv_bytes(before) + _STATE // 2     # the snapshot
    return {"bytes": b, "flops": f}


def tolerance(case):
    kind = case["kind"]
    if kind == "gemv":
        # many tokens of IQ3_S: f16 weights with one rounding each; else exact weights against 22-bit activations, f32 sums
        return {"rel": 1e-3} if case["type"] == "IQ3_S" and case["t"] >= 32 else {"rel": 1e-5}
    if kind == "decode":
        return "exact"     # token ids
    if kind == "prompt":
        return {"rel": 5e-3}     # f16 weights in the projections, through four layers and the recurrence
    return {"rel": 1e-4, "differ": 0.01}     # f32 sums through a block or four layers; expert ids may differ in a tie
