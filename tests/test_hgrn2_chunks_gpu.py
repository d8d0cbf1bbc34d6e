"""The HGRN2 recurrence in chunks of 64 tokens side by side, against float64 and against the walk token by token."""
import numpy as np
import pytest
import torch

import plain_fanidra as pf
from test_fanidra_gpu import TD, Step, bf16_round, dev

pytestmark = pytest.mark.gpu


def projections(T, H, d, dv, seed, gates):
    rng = np.random.default_rng(seed)
    zq, zf, v = (bf16_round(rng.normal(size=(T, H * n))) for n in (d, d, dv))
    if gates == "slow":
        zf = bf16_round(zf * 3 + 2)                      # near one: the state remembers far back
    elif gates == "all or nothing":
        zf = bf16_round(np.where(zf > 0, 200.0, -200.0))   # exactly one and (almost) zero: nothing may overflow
    lower = np.zeros(H * d) if gates == "all or nothing" else rng.uniform(0, 0.9, size=H * d)
    return np.concatenate([zq, zf, v], axis=1), rng.normal(size=H * d) * 0.1, lower, 1 + 0.1 * rng.normal(size=dv)


def scan(proj, lens, starts, H, d, dv, f_bias, lower, norm_w, state, dtype, chunks, monkeypatch, slots, pad=3):
    """One step over the requests' next ``lens`` tokens from ``starts``; proj: per request.  -> rows per request.
    chunks: True all in chunks, False none, None each by its own portion."""
    from swifttransformer_b200 import ops
    monkeypatch.setattr(ops, "HGRN2_CHUNK_MIN_TOKENS", {True: 1, False: 1 << 30, None: 96}[chunks])
    st = Step([(s, a, n) for s, a, n in zip(slots, starts, lens)], pad_tokens=pad, pad_requests=2)
    rows = np.concatenate([p[a:a + n] for p, a, n in zip(proj, starts, lens)] + [np.full((pad, proj[0].shape[1]), 50.0)])
    rows = dev(rows, TD[dtype])
    out = torch.full((st.n_rows, H * dv), 77.0, dtype=TD[dtype], device="cuda")
    need = int(ops.lib().st_hgrn2_chunks_scratch(st.n_rows, st.n_seqs, H, d, dv))
    scratch = torch.full((max(need, st.n_rows * H * dv),), float("nan"), device="cuda")
    split = ops.hgrn2_split(lens, st.n_rows, st.n_seqs, H, d) if chunks is None else None
    assert need > 0 and (not chunks or ops._hgrn2_chunks_apply(st.n_rows, st.n_seqs, H, d, dv, scratch, (rows.shape[1], 0, H * d, 2 * H * d),
                                                               (rows, out, state)))
    ops.hgrn2_scan(rows, 0, H * d, 2 * H * d, dev(f_bias), dev(lower), dev(norm_w), 1e-5, state, out, st.positions,
                   st.q_start, st.slots, st.n_seqs, H, d, dv, scratch=scratch, split=split)
    assert torch.all(out[st.n:] == 77.0)
    o, at, res = out.double().cpu().numpy(), 0, []
    for n in lens:
        res.append(o[at:at + n])
        at += n
    return res


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("gates", ["slow", "fast", "all or nothing"])
@pytest.mark.parametrize("H,d,dv", [(2, 128, 128), (3, 64, 36), (1, 4, 128), (2, 100, 4), (1, 36, 68)])
def test_chunks_in_portions(dtype, gates, H, d, dv, monkeypatch):
    # whole and in portions: one token, 31 to 33 (a half of a chunk), 63 to 65, several chunks and their edges, side by side
    lengths = [(64, 1, 130), (33, 200, 65), (31, 63, 32), (128, 2, 257)]
    total = [sum(n) for n in lengths]
    data = [projections(T, H, d, dv, 10 * i + d, gates) for i, T in enumerate(total)]
    f_bias, lower, norm_w = data[0][1:]
    proj = [x[0] for x in data]
    # (float32 inputs of the kernel: the reference starts from the same numbers)
    f_bias, lower, norm_w = (a.astype(np.float32).astype(np.float64) for a in (f_bias, lower, norm_w))
    refs = [pf.gated_recurrence(p[:, :H * d], p[:, H * d:2 * H * d], p[:, 2 * H * d:], f_bias, lower, norm_w, H, d, dv, 1e-5)
            for p in proj]
    slots = [4, 1, 3, 2]
    for cuts in (None, lengths):
        state = torch.zeros((5, H, d, dv), device="cuda")
        state[0].fill_(3.0)
        walked = state.clone()
        steps = [list(total)] if cuts is None else [[n[k] for n in cuts] for k in range(3)]
        at = [0] * 4
        for lens in steps:
            got = scan(proj, lens, at, H, d, dv, f_bias, lower, norm_w, state, dtype, True, monkeypatch, slots)
            scan(proj, lens, at, H, d, dv, f_bias, lower, norm_w, walked, dtype, False, monkeypatch, slots)
            for g, r, a, n in zip(got, refs, at, lens):
                # the bounds the walk is held to
                assert np.abs(g - r[a:a + n]).max() < (2e-5 if dtype == "float32" else 3e-2) * np.abs(r).max()
            at = [a + n for a, n in zip(at, lens)]
        assert torch.all(state[0] == 3.0) and torch.isfinite(state).all()
        assert (state - walked).abs().max() <= 4e-6 * walked[1:].abs().max()


def test_little_scratch_walks(monkeypatch):
    """Scratch that does not hold a state per chunk: the walk, as before."""
    from swifttransformer_b200 import ops
    H, d, dv, T = 2, 128, 128, 140
    p, f_bias, lower, norm_w = projections(T, H, d, dv, 1, "slow")
    st = Step([(1, 0, T)])
    outs = []
    for lim in (1, 1 << 30):
        monkeypatch.setattr(ops, "HGRN2_CHUNK_MIN_TOKENS", lim)
        out, state = torch.zeros((T, H * dv), device="cuda"), torch.zeros((2, H, d, dv), device="cuda")
        ops.hgrn2_scan(dev(p), 0, H * d, 2 * H * d, dev(f_bias), dev(lower), dev(norm_w), 1e-5, state, out, st.positions,
                       st.q_start, st.slots, 1, H, d, dv, scratch=torch.zeros(T * H * dv, device="cuda"))
        outs.append(out)
    assert torch.equal(*outs)


@pytest.mark.parametrize("t0", [1, 15, 16, 31, 40, 63, 64, 100])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_a_broken_token_leaves_the_ones_before_it(t0, bad, monkeypatch):
    """A value, a query or a gate that is not finite: the tokens before it, and the other heads, keep their numbers."""
    H, d, dv, T = 2, 64, 36, 150
    p, f_bias, lower, norm_w = projections(T, H, d, dv, t0, "slow")
    for col in (2 * H * d + 3, 5, H * d + 7):            # of head 0: a value, a query, a gate
        outs = []
        for x in (p[t0, col], bad):
            q = p.copy()
            q[t0, col] = x
            state = torch.zeros((2, H, d, dv), device="cuda")
            outs.append(scan([q], [T], [0], H, d, dv, f_bias, lower, norm_w, state, "float32", True, monkeypatch, [1])[0])
        assert np.array_equal(outs[0][:t0], outs[1][:t0]) and np.array_equal(outs[0][:, dv:], outs[1][:, dv:])


def test_each_request_goes_by_its_own_portion(monkeypatch):
    """Long portions beside single tokens and short ones: every request has the numbers of its own form."""
    H, d, dv = 2, 128, 36
    lens = [1, 300, 1, 95, 96, 130, 1, 64]
    data = [projections(n, H, d, dv, i, "slow") for i, n in enumerate(lens)]
    proj, (f_bias, lower, norm_w) = [x[0] for x in data], data[0][1:]
    slots, outs, states = [3, 1, 4, 8, 5, 2, 6, 7], [], []
    for chunks in (None, True, False):
        state = torch.linspace(-1, 1, 9 * H * d * dv, device="cuda").view(9, H, d, dv).contiguous()
        outs.append(scan(proj, lens, [0] * 8, H, d, dv, f_bias, lower, norm_w, state, "float32", chunks, monkeypatch, slots))
        states.append(state)
    for i, (n, s) in enumerate(zip(lens, slots)):
        k = 1 if n >= 96 else 2
        assert np.array_equal(outs[0][i], outs[k][i]) and torch.equal(states[0][s], states[k][s])
    # alone in its step, the long one has the same numbers
    state = torch.linspace(-1, 1, 9 * H * d * dv, device="cuda").view(9, H, d, dv).contiguous()
    lone = scan(proj[1:2], [300], [0], H, d, dv, f_bias, lower, norm_w, state, "float32", None, monkeypatch, [1], pad=20)
    assert np.array_equal(lone[0], outs[0][1]) and torch.equal(state[1], states[0][1])
