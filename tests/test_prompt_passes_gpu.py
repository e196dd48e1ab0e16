"""Prompt passes and the kernels that only they and large batches reach: runs of the DeltaNet recurrence in blocks of eight tokens, the router and its lists for many tokens,
several prompt chunks in one pass, expert groups of up to 24 entries."""
import os

import numpy as np
import pytest

import pyre_b200 as pb
from pyre_b200 import synth
from conftest import rel_err
from helpers import oracle_cfg, oracle_model, small_cfg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16, 23, 24, 31, 32, 39, 40])
def test_deltanet_blocks_of_tokens(ctx, n):
    """The longest run token by token, full blocks of eight (from 32 tokens on) and a last block of seven: the state that n single steps leave (Q4_K: exact
    weights in the projections; two layers and the gates amplify the last bits of f32 sums)."""
    cfg = small_cfg(pb, n_layers=2, full_every=0)
    m = synth.build_model(ctx, cfg, synth.model_spec(cfg, 9, pb.Q4_K), 9)
    a, b = m.new_state(1), m.new_state(1)
    ids = np.random.default_rng(n).integers(0, cfg.vocab, n).astype(np.uint32)
    la = a.forward(ids)
    for t in ids:
        lb = b.forward(np.array([t], np.uint32))
    assert rel_err(la, lb) < 1e-4
    for (ca, sa), (cb, sb) in zip((a.get_lin(0), a.get_lin(1)), (b.get_lin(0), b.get_lin(1))):
        assert rel_err(ca, cb) < 1e-4 and rel_err(sa, sb) < 1e-4
    assert ctx.device_status() == 0
    a.destroy(); b.destroy(); m.destroy()


@pytest.mark.parametrize("t", [128, 131, 261])
def test_router_of_many_tokens(ctx, t):
    """70 experts (a ragged last group of router rows), the last group of tokens full and ragged: selection and block
    against the oracle; the first tokens' results are those of a call of two tokens, bit for bit."""
    import oracle
    cfg = small_cfg(pb, n_layers=1, full_every=0, d=2048, n_exp=70)
    spec = synth.model_spec(cfg, 6)
    m = synth.build_model(ctx, cfg, spec, 6)
    _, mats = oracle_model(cfg, spec, 6)
    st = m.new_state(t)
    x = np.random.default_rng(t).standard_normal((t, cfg.d)).astype(np.float32)
    y, sel = st.moe_forward(0, x)
    yo, selo, _ = oracle.moe(oracle_cfg(cfg), *(mats[(0, r)] for r in ("ROUTER", "EXP_GATE", "EXP_UP", "EXP_DOWN", "SH_GATE", "SH_UP", "SH_DOWN", "SH_GATE_INP")), x)
    assert np.array_equal(np.sort(sel, axis=1), np.sort(selo, axis=1))
    assert rel_err(y, yo) < 1e-5
    y1, _ = st.moe_forward(0, x[:2])
    assert np.array_equal(y1.view(np.uint32), y[:2].view(np.uint32))
    assert ctx.device_status() == 0
    st.destroy(); m.destroy()


@pytest.mark.parametrize("n", [272, 1024, 1295, 1313])
def test_several_chunks_in_one_pass(ctx, n):
    """Whole chunks and a rest of 0, 15 (a pass of its own), 16 and 33 tokens: logits, states and the tokens that follow are those of a call per chunk, bit for bit."""
    cfg = small_cfg(pb, max_ctx=1400, kv_bits=4)
    m = synth.build_model(ctx, cfg, synth.model_spec(cfg, 12), 12)
    a, b = m.new_state(1), m.new_state(1)
    ids = np.random.default_rng(n).integers(0, cfg.vocab, n).astype(np.uint32)
    la = a.forward(ids)
    for i in range(0, n, 256):
        lb = b.forward(ids[i:i + 256])
    assert np.array_equal(la.view(np.uint32), lb.view(np.uint32))
    for (ca, sa), (cb, sb) in zip((a.get_lin(0), a.get_lin(2)), (b.get_lin(0), b.get_lin(2))):
        assert np.array_equal(ca.view(np.uint32), cb.view(np.uint32)) and np.array_equal(sa.view(np.uint32), sb.view(np.uint32))
    assert a.decode_greedy([5], 8)[0].tolist() == b.decode_greedy([5], 8)[0].tolist()
    assert ctx.device_status() == 0
    a.destroy(); b.destroy(); m.destroy()


@pytest.mark.parametrize("name,start,kw", [
    ("Q4_K", 0, dict(kv_bits=4)),                              # projections in launches of 32, experts at the warp level
    ("IQ3_S", 0, dict(kv_bits=0)),                             # f32 cache
    ("IQ3_S", 40, dict(kv_bits=4)),                            # off the grid: a piece up to the next multiple of 256 goes first
    ("IQ3_S", 256, dict(kv_bits=4)),                           # on it
    ("IQ3_S", 0, dict(kv_bits=4, full_every=2, n_rot=32)),     # attention without the shared tiles, two layers of it
    ("IQ3_S", 0, dict(kv_bits=4, lin_dk=64)),                  # no blocks of tokens in the recurrence
])
@pytest.mark.parametrize("n", [560, 600, 1060])
def test_several_chunks_in_one_pass_of_other_models_and_starts(ctx, name, start, kw, n):
    """Two to four chunks and a rest of 36 to 88 tokens: one call with passes over several chunks against one with a pass per chunk.  That the first call
    has such passes shows in the memory of their row buffers, which turning them off gives back."""
    import torch
    cfg = small_cfg(pb, max_ctx=1400, **kw)
    m = synth.build_model(ctx, cfg, synth.model_spec(cfg, 12, getattr(pb, name)), 12)
    rng = np.random.default_rng(n)
    before, ids = rng.integers(0, cfg.vocab, 256).astype(np.uint32)[:start], rng.integers(0, cfg.vocab, n).astype(np.uint32)
    got = []
    a, b = m.new_state(1), m.new_state(1)
    for st in (a, b):
        if start:
            st.forward(before)
        if st is b:
            ctx.sync(); free = torch.cuda.mem_get_info(0)[0]
            m.prompt_passes(False)
            if name != "IQ3_S" or os.environ.get("PYRE_B200_REPACK") != "0":       # (without re-coded copies IQ3_S has no experts on the tensor cores, and no such passes)
                assert torch.cuda.mem_get_info(0)[0] >= free + (16 << 20)
        lg = st.forward(ids)
        got.append((lg, *[x for il in range(cfg.n_layers) if (il + 1) % cfg.full_every for x in st.get_lin(il)], st.decode_greedy([5], 8)))
    for u, v in zip(*got):
        assert np.array_equal(np.asarray(u).view(np.uint32), np.asarray(v).view(np.uint32))
    assert ctx.device_status() == 0
    a.destroy(); b.destroy(); m.destroy()


@pytest.mark.parametrize("t", [31, 32, 97, 161])
def test_expert_groups_of_many_entries(ctx, t):
    """16 experts, 4 per token: around the number of tokens from which the tcgen05 kernels take over, and groups of up to 24 entries with ragged ends; the
    first tokens' results are those of a call of two tokens, bit for bit."""
    import oracle
    cfg = small_cfg(pb, n_layers=1, full_every=0)
    spec = synth.model_spec(cfg, 8)
    m = synth.build_model(ctx, cfg, spec, 8)
    _, mats = oracle_model(cfg, spec, 8)
    st = m.new_state(t)
    x = np.random.default_rng(t).standard_normal((t, cfg.d)).astype(np.float32)
    y, sel = st.moe_forward(0, x)
    yo, selo, _ = oracle.moe(oracle_cfg(cfg), *(mats[(0, r)] for r in ("ROUTER", "EXP_GATE", "EXP_UP", "EXP_DOWN", "SH_GATE", "SH_UP", "SH_DOWN", "SH_GATE_INP")), x)
    assert np.array_equal(np.sort(sel, axis=1), np.sort(selo, axis=1))
    assert rel_err(y, yo) < 1e-5
    for i in range(0, t - 1, 2):
        y1, _ = st.moe_forward(0, x[i:i + 2])
        assert np.array_equal(y1.view(np.uint32), y[i:i + 2].view(np.uint32)), i
    assert ctx.device_status() == 0
    st.destroy(); m.destroy()
