"""The warp-level tensor-core kernels (several tokens against quantized weights) at the edges of their tiles: rows around the 16-row tile and the
eight-row group of the re-coded form, one to sixteen blocks per row (a cluster of CTAs above eight), token counts around the n-tiles of
four and the sixteen of a launch; expert groups around eight entries; runs of the DeltaNet recurrence around their blocks of tokens."""
import numpy as np
import pytest

import oracle
import pyre_b200 as pb
from pyre_b200 import synth
from conftest import rel_err
from helpers import oracle_cfg, oracle_model, small_cfg

pytestmark = pytest.mark.gpu
TOL = 3e-6   # f32 sums of exact weights against 22-bit activations


@pytest.mark.parametrize("name", ["IQ3_S", "Q4_K", "IQ2_XS", "Q8_0", "Q5_K", "Q6_K"])
@pytest.mark.parametrize("rows,cols", [(1, 256), (17, 512), (515, 2048), (40, 4096), (2400, 1024)])
def test_gemm_tile_edges(ctx, name, rows, cols):
    ty = getattr(pb, name)
    W, Wo = pb.QMat.synth(ctx, ty, rows, cols, 0, 77), oracle.QMat.synth(ty, rows, cols, 0, 77)
    rng = np.random.default_rng(rows + cols)
    x = rng.standard_normal((19, cols)).astype(np.float32)
    x[1, :128] *= 1e4; x[2] *= 1e-5; x[3, cols // 2:] = 0.0
    ref = Wo.matmul(x)
    scale = np.linalg.norm(x, axis=1) * np.linalg.norm(Wo.to_f32(), axis=1).max()   # a single row may cancel: relative to its operands
    for t in (2, 4, 5, 8, 9, 16, 17, 19):
        y = W.matmul(x[:t])
        for b in range(t):
            assert np.abs(y[b] - ref[b]).max() <= TOL * scale[b], (t, b)
    assert ctx.device_status() == 0
    W.free()


@pytest.mark.parametrize("name", ["IQ3_S", "Q4_K"])
@pytest.mark.parametrize("t", [2, 5, 33, 70])
def test_expert_groups_of_more_and_fewer_than_eight_entries(ctx, name, t):
    """16 experts, 4 per token: from one entry per expert to several groups of eight, the last one ragged."""
    cfg = small_cfg(pb, n_layers=1, full_every=0)
    spec = synth.model_spec(cfg, 5, qtype=getattr(pb, name))
    m = synth.build_model(ctx, cfg, spec, 5)
    _, mats = oracle_model(cfg, spec, 5)
    st = m.new_state(t)
    x = np.random.default_rng(t).standard_normal((t, cfg.d)).astype(np.float32)
    y, sel = st.moe_forward(0, x)
    yo, selo, _ = oracle.moe(oracle_cfg(cfg), *(mats[(0, r)] for r in ("ROUTER", "EXP_GATE", "EXP_UP", "EXP_DOWN", "SH_GATE", "SH_UP", "SH_DOWN", "SH_GATE_INP")), x)
    assert np.array_equal(np.sort(sel, axis=1), np.sort(selo, axis=1))
    assert rel_err(y, yo) < 1e-5
    y1, _ = st.moe_forward(0, x[:2])           # a token's result does not depend on the tokens beside it
    assert t == 2 or np.array_equal(y1.view(np.uint32), y[:2].view(np.uint32))
    assert ctx.device_status() == 0
    st.destroy(); m.destroy()


@pytest.mark.parametrize("n", [3, 8, 9, 31, 33])
def test_deltanet_run_lengths(ctx, n):
    """A prompt of n tokens (one run of the recurrence) leaves the state that n single steps leave."""
    cfg = small_cfg(pb, n_layers=2, full_every=0)
    m = synth.build_model(ctx, cfg, synth.model_spec(cfg, 9), 9)
    a, b = m.new_state(1), m.new_state(1)
    ids = np.random.default_rng(n).integers(0, cfg.vocab, n).astype(np.uint32)
    la = a.forward(ids)
    for t in ids:
        lb = b.forward(np.array([t], np.uint32))
    tol = 1e-4 if n < 16 else 5e-3             # two layers and the gates amplify the last bits; from 16 tokens on the projections' weights are rounded to f16
    assert rel_err(la, lb) < tol
    for (ca, sa), (cb, sb) in zip((a.get_lin(0), a.get_lin(1)), (b.get_lin(0), b.get_lin(1))):
        assert rel_err(ca, cb) < tol and rel_err(sa, sb) < tol
    a.destroy(); b.destroy(); m.destroy()


@pytest.mark.parametrize("n_head,n_kv", [(4, 2), (8, 1), (2, 2)])
@pytest.mark.parametrize("prefix,t", [(0, 3), (60, 9), (127, 15), (250, 7), (383, 12)])
def test_window_attention_matches_single_steps(ctx, n_head, n_kv, prefix, t):
    """Windows whose tokens straddle the 64-position tiles and the boundary of the packed cache, one to three of which fill a row tile
    (t < 16: the projections keep exact weights), then single steps over what the window left in the cache."""
    cfg = small_cfg(pb, n_layers=2, full_every=1, n_head=n_head, n_kv=n_kv, kv_bits=4, kv_recent=64)
    m = synth.build_model(ctx, cfg, synth.model_spec(cfg, 11), 11)
    a, b = m.new_state(1), m.new_state(1)
    ids = np.random.default_rng(prefix + t).integers(0, cfg.vocab, t).astype(np.uint32)
    for s in (a, b):
        if prefix:
            for ai in range(2):
                s.fill_kv_synth(ai, prefix, 3)
            s.set_pos(prefix)
    la = a.forward(ids)
    for i in ids:
        lb = b.forward(np.array([i], np.uint32))
    assert rel_err(la, lb) < 1e-4
    for _ in range(3):
        assert rel_err(a.forward(ids[:1]), b.forward(ids[:1])) < 1e-3    # a rounding of a value may fall the other way in the packed cache
    assert ctx.device_status() == 0
    a.destroy(); b.destroy(); m.destroy()
