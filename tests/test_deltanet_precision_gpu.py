"""Runs of the DeltaNet recurrence against 64 bits, from their own f32 projections: the blocks of eight tokens that prompts of 32 and more tokens take must be no
farther off than the walk token by token, which the same tokens take in pieces of eight; and a token that is not finite must not reach the tokens before it."""
import numpy as np
import pytest

import oracle
import pyre_b200 as pb
from pyre_b200 import synth
from pyre_b200.model import Model
from helpers import small_cfg

pytestmark = pytest.mark.gpu


def _cfg():
    return small_cfg(pb, n_layers=1, full_every=0, lin_nk=16, lin_nv=32)


def _ld(cfg):
    return (max(2 * cfg.lin_nk * cfg.lin_dk + 2 * cfg.lin_nv * cfg.lin_dv + 2 * cfg.lin_nv, 2 * cfg.n_head * cfg.hd + 2 * cfg.n_kv * cfg.hd) + 3) // 4 * 4


def _f64(cfg, spec, proj):
    """Readout and state after the tokens whose projections [qkv | z | beta | alpha] are given (linear_core, src/model/qwen4exp_gguf.rs:1624-1666)."""
    vec = {s[2]: s[3].astype(np.float64) for s in spec if s[0] == "vec" and s[1] == 0}
    nk, nv, dk, dv, n = cfg.lin_nk, cfg.lin_nv, cfg.lin_dk, cfg.lin_dv, len(proj)
    ch, p = 2 * nk * dk + nv * dv, proj.astype(np.float64)
    beta, alpha = p[:, ch + nv * dv:ch + nv * dv + nv], p[:, ch + nv * dv + nv:ch + nv * dv + 2 * nv]
    w, h = vec["LIN_CONV"].reshape(-1, cfg.conv_k), np.vstack([np.zeros((cfg.conv_k - 1, ch)), p[:, :ch]])
    o = sum(h[i:i + n] * w[:, i] for i in range(cfg.conv_k))
    sig = lambda x: 0.5 * (1.0 + np.tanh(0.5 * x))
    o *= sig(o)
    q, k, v = o[:, :nk * dk].reshape(n, nk, dk), o[:, nk * dk:2 * nk * dk].reshape(n, nk, dk), o[:, 2 * nk * dk:].reshape(n, nv, dv)
    q = q / np.sqrt((q * q).sum(-1, keepdims=True) + 1e-6) / np.sqrt(dk)
    k = k / np.sqrt((k * k).sum(-1, keepdims=True) + 1e-6)
    g, b = np.exp(np.logaddexp(0.0, alpha + vec["LIN_DT"]) * vec["LIN_A"]), sig(beta)
    S, out, idx = np.zeros((nv, dk, dv)), np.empty((n, nv, dv)), np.arange(nv) % nk
    for t in range(n):
        kk, qq = k[t, idx], q[t, idx]
        S *= g[t][:, None, None]
        S += kk[:, :, None] * ((v[t] - np.einsum("hij,hi->hj", S, kk)) * b[t][:, None])[:, None]
        out[t] = np.einsum("hij,hi->hj", S, qq)
    return out, S


@pytest.mark.parametrize("decay", [1.0, 1e-3, 30.0])          # as synthesised; near 1, where the state of hundreds of tokens ago counts; near 0
@pytest.mark.parametrize("n", [32, 39, 256])
def test_blocks_are_as_close_to_64_bits_as_single_tokens(ctx, n, decay):
    """The bound: the walk's own error in the mean of three models; 3 % for the state, whose rounding differs in order only."""
    cfg = _cfg()
    err = np.zeros((3, 2, 2))
    for seed in range(3):
        spec = [s if s[2] != "LIN_A" else (*s[:3], (s[3] * decay).astype(np.float32)) for s in synth.model_spec(cfg, seed, pb.Q4_K)]   # (exact weights in projections of any number of tokens: both ways see the same ones)
        m = synth.build_model(ctx, cfg, spec, seed)
        ids = np.random.default_rng(seed).integers(0, cfg.vocab, n).astype(np.uint32)
        for i, step in enumerate((n, 8)):
            st = m.new_state(1)
            proj, out = [], []
            for t0 in range(0, n, step):
                k = min(step, n - t0)
                st.forward(ids[t0:t0 + k])
                proj.append(st.peek(1, k * _ld(cfg)).reshape(k, -1))
                out.append(st.peek(2, k * cfg.lin_nv * cfg.lin_dv).reshape(k, cfg.lin_nv, cfg.lin_dv))
            ro, rs = _f64(cfg, spec, np.concatenate(proj))
            S = np.asarray(st.get_lin(0)[1], np.float64).reshape(rs.shape)
            err[seed, i] = np.linalg.norm(np.concatenate(out) - ro) / np.linalg.norm(ro), np.linalg.norm(S - rs) / np.linalg.norm(rs)
            st.destroy()
        m.destroy()
    (out_b, state_b), (out_w, state_w) = err.mean(axis=0)
    print(f"n {n} decay {decay}: readout {out_b:.3e} / {out_w:.3e}, state {state_b:.3e} / {state_w:.3e}")
    assert out_b <= out_w and state_b <= 1.03 * state_w
    assert out_w < 2e-7 and state_w < 4e-7
    assert ctx.device_status() == 0


@pytest.mark.parametrize("bad_at", [0, 7, 8, 13, 38])
def test_a_token_that_is_not_finite_leaves_the_readout_before_it_alone(ctx, bad_at):
    cfg = _cfg()
    spec, bad = synth.model_spec(cfg, 13), 77
    m = Model(ctx, cfg)
    for item in spec:
        if item[0] == "vec":
            m.set_vec(item[1], item[2], item[3])
        elif item[2] == "TOKEN_EMBD":
            emb = oracle.synth_normal(13, item[6], 0, item[4] * item[5], 0.02).reshape(item[4], item[5])
            emb[bad, 3] = np.nan
            m.set_tensor(-1, "TOKEN_EMBD", pb.QMat.upload(ctx, pb.F32, item[4], item[5], emb))
        else:
            m.set_tensor(item[1], item[2], pb.QMat.synth(ctx, item[3], item[4], item[5], 13, item[6]))
    m.finalize()
    st = m.new_state(1)
    out = []
    for tok in (bad, 5):
        st.reset()
        ids = np.arange(100, 139, dtype=np.uint32)
        ids[bad_at] = tok
        st.forward(ids)
        out.append(st.peek(2, 39 * cfg.lin_nv * cfg.lin_dv).reshape(39, -1))
    assert np.array_equal(out[0][:bad_at].view(np.uint32), out[1][:bad_at].view(np.uint32))
    assert np.isnan(out[0][bad_at:]).all() and np.isfinite(out[1]).all()
    assert ctx.device_status() == 0
    st.destroy(); m.destroy()
