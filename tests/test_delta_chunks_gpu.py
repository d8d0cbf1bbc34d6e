"""The gated delta rule in chunks of 64 tokens side by side, against float64 and against the walk token by token."""
import numpy as np
import pytest
import torch

import plain_norelix as pn
from test_fanidra_gpu import TD, Step, dev

pytestmark = pytest.mark.gpu


def inputs(T, H, G, d, dv, rank, seed, decays, same_keys=False):
    """Float32 projections of one request and the mixer's small weights (float64 arrays of float32 values)."""
    rng = np.random.default_rng(seed)
    f32 = lambda a: np.asarray(a, dtype=np.float32).astype(np.float64)
    bf = lambda a: torch.tensor(a, dtype=torch.float32).to(torch.bfloat16).double().numpy()
    C = 2 * G * d + H * dv
    cols = C + H + (2 * rank if rank else H + H * dv)
    proj = rng.normal(size=(T, cols))
    if same_keys:                                    # every key the same one: the corrections between tokens are largest
        proj[:, G * d:2 * G * d] = proj[0, G * d:2 * G * d]
        proj[:, C:C + H] = 8.0                       # write strengths near one
    w = dict(conv=f32(rng.normal(size=(C, 2)) * 0.6), norm=f32(1 + 0.2 * rng.normal(size=dv)),
             A_log=f32(np.full(H, {"slow": -6.0, "fast": 2.0, "none": -300.0, "all": 6.0}[decays])))
    if same_keys:
        w["conv"][:, 0] = 0.0
    w["dt_bias"] = f32(rng.normal(size=H * d if rank else H) * 0.5)
    w["a2"], w["g2"] = (bf(rng.normal(size=(H * d, rank)) * 0.5), bf(rng.normal(size=(H * dv, rank)) * 0.5)) if rank else (None, None)
    return f32(proj), w


def reference(proj, w, H, G, d, dv, rank, eps, out_scale):
    T, C = len(proj), 2 * G * d + H * dv
    past = np.concatenate([np.zeros((1, C)), proj[:, :C]])
    z = past[:-1] * w["conv"][:, 0] + past[1:] * w["conv"][:, 1]
    z = z * pn.sigmoid(z)
    q, k, v = z[:, :G * d].reshape(T, G, d), z[:, G * d:2 * G * d].reshape(T, G, d), z[:, 2 * G * d:].reshape(T, H, dv)
    q = q / np.sqrt((q * q).sum(-1, keepdims=True) + 1e-6) * d ** -0.5
    k = k / np.sqrt((k * k).sum(-1, keepdims=True) + 1e-6)
    beta = pn.sigmoid(proj[:, C:C + H])
    if rank:
        dt, gate = proj[:, C + H:C + H + rank] @ w["a2"].T + w["dt_bias"], proj[:, C + H + rank:] @ w["g2"].T
    else:
        dt, gate = np.repeat(proj[:, C + H:C + 2 * H] + w["dt_bias"], d, axis=1), proj[:, C + 2 * H:]
    decay = np.exp(-np.exp(w["A_log"])[:, None] * np.logaddexp(dt, 0).reshape(T, H, d))
    o, S = np.zeros((T, H, dv)), np.zeros((H, d, dv))
    for t in range(T):
        for h in range(H):
            g = h // (H // G)
            S[h] *= decay[t, h][:, None]
            S[h] += np.outer(k[t, g], beta[t, h] * (v[t, h] - k[t, g] @ S[h]))
            o[t, h] = q[t, g] @ S[h]
    o = o / np.sqrt((o * o).mean(-1, keepdims=True) + eps) * w["norm"] * out_scale
    return o.reshape(T, H * dv) * pn.sigmoid(gate), S


def step(projs, lens, starts, H, G, d, dv, rank, w, tails, state, dtype, chunks, monkeypatch, slots, write=True, pad=3):
    """One step over the requests' next tokens; -> rows per request.  chunks: True all in chunks, False none, None
    each by its own portion."""
    from swifttransformer_b200 import ops
    monkeypatch.setattr(ops, "DELTA_CHUNK_MIN_TOKENS", {True: 1, False: 1 << 30, None: 256}[chunks])
    st = Step([(s, a, n) for s, a, n in zip(slots, starts, lens)], pad_tokens=pad, pad_requests=2)
    rows = dev(np.concatenate([p[a:a + n] for p, a, n in zip(projs, starts, lens)] + [np.full((pad, projs[0].shape[1]), 7.0)]))
    C = 2 * G * d + H * dv
    need = int(ops.lib().st_delta_rule_chunk_floats(st.n_rows, st.n_seqs, H, G, d, dv))
    assert need > 0
    scratch = torch.full((max(need, ops.delta_rule_scratch(st.n_rows, H, G, d, dv)),), float("nan"), device="cuda")
    out = torch.full((st.n_rows, H * dv), 77.0, dtype=TD[dtype], device="cuda")
    low = lambda a: None if a is None else dev(a, TD[dtype])
    split = ops.delta_split(lens, st.n_rows, st.n_seqs) if chunks is None else None
    ops.delta_rule(rows, C, C + H, C + H + (rank or H), dev(w["conv"]), tails, low(w["a2"]), dev(w["A_log"]), dev(w["dt_bias"]),
                   low(w["g2"]), dev(w["norm"]), 1e-5, 0.7, state, write, False, scratch, out, st.positions, st.seq, st.q_start,
                   st.slots, st.n_seqs, H, G, d, dv, split=split)
    ops.conv_state_update(rows, C, tails, st.positions, st.q_start, st.slots, st.n_seqs)
    assert torch.all(out[st.n:] == 77.0)
    o, at, res = out.double().cpu().numpy(), 0, []
    for n in lens:
        res.append(o[at:at + n])
        at += n
    return res


SHAPES = [(4, 2, 128, 128, 16), (2, 2, 64, 36, 0), (3, 1, 100, 4, 5), (1, 1, 4, 128, 8), (16, 8, 36, 68, 0)]


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("decays", ["slow", "fast", "none", "all"])
@pytest.mark.parametrize("H,G,d,dv,rank", SHAPES)
def test_chunks_in_portions(dtype, decays, H, G, d, dv, rank, monkeypatch):
    # whole and in portions: one token, 31 to 33 (a half of a chunk), 63 to 65, several chunks and their edges, side by side
    lengths = [(64, 1, 130), (33, 200, 65), (31, 63, 32), (128, 2, 257)]
    total = [sum(n) for n in lengths]
    projs = [inputs(T, H, G, d, dv, rank, 10 * i + d, decays)[0] for i, T in enumerate(total)]
    w = inputs(1, H, G, d, dv, rank, d, decays)[1]
    refs = [reference(p, w, H, G, d, dv, rank, 1e-5, 0.7) for p in projs]
    slots, C = [4, 1, 3, 2], 2 * G * d + H * dv
    for cuts in (None, lengths):
        state, tails = torch.zeros((5, H, d, dv), device="cuda"), torch.zeros((5, 1, C), device="cuda")
        state[0].fill_(3.0)
        steps = [list(total)] if cuts is None else [[n[k] for n in cuts] for k in range(3)]
        at = [0] * 4
        for lens in steps:
            got = step(projs, lens, at, H, G, d, dv, rank, w, tails, state, dtype, True, monkeypatch, slots)
            for g, (r, _), a, n in zip(got, refs, at, lens):
                # the bounds the walk is held to
                assert np.abs(g - r[a:a + n]).max() < (3e-5 if dtype == "float32" else 3e-2) * np.abs(r).max()
            at = [a + n for a, n in zip(at, lens)]
        assert torch.all(state[0] == 3.0)
        for s, (_, S) in zip(slots, refs):
            assert np.abs(state[s].double().cpu().numpy() - S).max() < 1e-5 * max(np.abs(S).max(), 1e-3)


def test_one_key_written_over_and_over(monkeypatch):
    """Every token writes the same key with a strength near one and nothing decays: each u takes back the one before."""
    H, G, d, dv, rank, T = 2, 1, 128, 64, 0, 300
    proj, w = inputs(T, H, G, d, dv, rank, 3, "none", same_keys=True)
    ref, S = reference(proj, w, H, G, d, dv, rank, 1e-5, 0.7)
    for write in (True, False):
        state, tails = torch.zeros((2, H, d, dv), device="cuda"), torch.zeros((2, 1, 2 * G * d + H * dv), device="cuda")
        got = step([proj], [T], [0], H, G, d, dv, rank, w, tails, state, "float32", True, monkeypatch, [1], write=write)[0]
        assert np.abs(got - ref).max() < 3e-5 * np.abs(ref).max()
        assert np.abs(state[1].double().cpu().numpy() - (S if write else 0 * S)).max() < 1e-5 * np.abs(S).max()


def test_little_scratch_walks(monkeypatch):
    """Scratch of the walk's size: the walk, as before."""
    from swifttransformer_b200 import ops
    H, G, d, dv, rank, T = 2, 2, 64, 64, 0, 300
    proj, w = inputs(T, H, G, d, dv, rank, 5, "slow")
    C, st, outs = 2 * G * d + H * dv, Step([(0, 0, T)]), []
    for lim in (1, 1 << 30):
        monkeypatch.setattr(ops, "DELTA_CHUNK_MIN_TOKENS", lim)
        out, state = torch.zeros((T, H * dv), device="cuda"), torch.zeros((1, H, d, dv), device="cuda")
        scratch = torch.zeros(int(ops.lib().st_delta_rule_scratch_floats(T, H, G, d, dv)), device="cuda")
        ops.delta_rule(dev(proj), C, C + H, C + 2 * H, dev(w["conv"]), torch.zeros((1, 1, C), device="cuda"), None, dev(w["A_log"]),
                       dev(w["dt_bias"]), None, dev(w["norm"]), 1e-5, 1.0, state, True, False, scratch, out, st.positions, st.seq,
                       st.q_start, st.slots, 1, H, G, d, dv)
        outs.append(out)
    assert torch.equal(*outs)


@pytest.mark.parametrize("t0", [1, 15, 16, 31, 40, 63, 64, 100])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_a_broken_token_leaves_the_ones_before_it(t0, bad, monkeypatch):
    """A value, a query, a key, a write strength or a decay that is not finite: the tokens before it, and the other heads, keep
    their numbers."""
    H, G, d, dv, rank, T = 2, 2, 64, 36, 0, 150
    proj, w = inputs(T, H, G, d, dv, rank, t0, "slow")
    C = 2 * G * d + H * dv
    for col in (2 * G * d + 3, 5, G * d + 7, C, C + H):    # of head 0
        outs = []
        for x in (proj[t0, col], bad):
            p = proj.copy()
            p[t0, col] = x
            state, tails = torch.zeros((2, H, d, dv), device="cuda"), torch.zeros((2, 1, C), device="cuda")
            outs.append(step([p], [T], [0], H, G, d, dv, rank, w, tails, state, "float32", True, monkeypatch, [1])[0])
        assert np.array_equal(outs[0][:t0], outs[1][:t0]) and np.array_equal(outs[0][:, dv:], outs[1][:, dv:])


def test_each_request_goes_by_its_own_portion(monkeypatch):
    """Long portions beside single tokens and short ones: every request has the numbers of its own form."""
    H, G, d, dv, rank = 2, 1, 64, 36, 0
    lens = [1, 300, 1, 255, 256, 400, 2]
    projs, w = [inputs(n, H, G, d, dv, rank, i, "slow")[0] for i, n in enumerate(lens)], inputs(1, H, G, d, dv, rank, 1, "slow")[1]
    slots, outs, states, C = [3, 1, 4, 7, 5, 2, 6], [], [], 2 * G * d + H * dv
    for chunks in (None, True, False):
        state = torch.linspace(-1, 1, 8 * H * d * dv, device="cuda").view(8, H, d, dv).contiguous()
        outs.append(step(projs, lens, [0] * 7, H, G, d, dv, rank, w, torch.zeros((8, 1, C), device="cuda"), state, "float32", chunks,
                         monkeypatch, slots))
        states.append(state)
    for i, (n, s) in enumerate(zip(lens, slots)):
        k = 1 if n >= 256 else 2
        assert np.array_equal(outs[0][i], outs[k][i]) and torch.equal(states[0][s], states[k][s])
    state = torch.linspace(-1, 1, 8 * H * d * dv, device="cuda").view(8, H, d, dv).contiguous()
    lone = step(projs[5:6], [400], [0], H, G, d, dv, rank, w, torch.zeros((8, 1, C), device="cuda"), state, "float32", None,
                monkeypatch, [2], pad=20)
    assert np.array_equal(lone[0], outs[0][5]) and torch.equal(state[2], states[0][2])
