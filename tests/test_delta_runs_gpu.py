"""The delta rule's preparation and output by runs of tokens (steps of more than 128 tokens) against the forms of small steps, bit
for bit."""
import numpy as np
import pytest
import torch

from test_fanidra_gpu import TD, Step, dev

pytestmark = pytest.mark.gpu


# heads of whole and ragged warps, filters of two to four taps, the low-rank pairs of sixteen, of another rank and none; one to four values
# more than a run, requests that begin inside a run
@pytest.mark.parametrize("H,G,d,dv,rank,taps", [(2, 1, 128, 128, 16, 4), (8, 4, 64, 128, 16, 4), (3, 1, 20, 36, 5, 3), (4, 2, 100, 33, 0, 2),
                                                (17, 1, 32, 16, 16, 4)])
@pytest.mark.parametrize("dtype,silu", [("float32", False), ("bfloat16", True)])
def test_runs_give_the_bits_of_small_steps(H, G, d, dv, rank, taps, dtype, silu, monkeypatch):
    from swifttransformer_b200 import ops
    monkeypatch.setattr(ops, "DELTA_CHUNK_MIN_TOKENS", 1 << 30)              # (every request walks)
    rng = np.random.default_rng(H * d + taps)
    C = 2 * G * d + H * dv
    cols = C + H + (2 * rank if rank else H + H * dv)
    lens = [37, 100, 5, 61]
    projs = [rng.normal(size=(n, cols)) for n in lens]
    conv = dev(rng.normal(size=(C, taps)) * 0.5)
    low = lambda *s: dev(rng.normal(size=s) * 0.3, TD[dtype]) if rank else None
    a2, g2 = low(H * d, rank), low(H * dv, rank)
    a_log, norm = dev(rng.normal(size=H)), dev(1 + 0.1 * rng.normal(size=dv))
    dt_bias = dev(rng.normal(size=H * d if rank else H))
    tails0 = dev(rng.normal(size=(5, taps - 1, C)))

    def run(which, pad):
        st = Step([(i, 0, lens[i]) for i in which], pad_tokens=pad, pad_requests=0)
        rows = dev(np.concatenate([projs[i] for i in which] + [np.full((pad, cols), 7.0)]))
        state = torch.zeros((5, H, d, dv), device="cuda")
        scratch = torch.full((ops.delta_rule_scratch(st.n_rows, H, G, d, dv),), float("nan"), device="cuda")
        out = torch.full((st.n_rows, H * dv), 77.0, dtype=TD[dtype], device="cuda")
        ops.delta_rule(rows, C, C + H, C + H + (rank or H), conv, tails0.clone(), a2, a_log, dt_bias, g2, norm, 1e-5, 0.7, state, True,
                       False, scratch, out, st.positions, st.seq, st.q_start, st.slots, st.n_seqs, H, G, d, dv, gate_silu=silu)
        assert torch.all(out[st.n:] == 77.0)
        return out, state
    ops.delta_rule_set_lanes(8)                                               # (the walk's own choice goes by the number of requests)
    try:
        out, state = run([0, 1, 2, 3], 4)                                     # 207 tokens: runs
        at = 0
        for i, n in enumerate(lens):
            small, s = run([i], 1)
            assert torch.equal(small[:n], out[at:at + n]) and torch.equal(s[i], state[i]), i
            at += n
    finally:
        ops.delta_rule_set_lanes(0)


# Runs of sixteen and of eight tokens (sixteen where that gives four blocks for each of 148 multiprocessors, else eight or four): taps that
# pass from one group of four to the next, requests and padding that begin at any place of a run, last runs that are not full
@pytest.mark.parametrize("H,G,d,dv,rank,taps,total", [(17, 1, 32, 16, 16, 4, 1613), (17, 1, 32, 16, 16, 4, 821), (8, 4, 64, 128, 16, 3, 2379),
                                                      (8, 4, 64, 128, 16, 2, 1203), (4, 2, 100, 33, 0, 2, 3167), (3, 1, 20, 36, 5, 4, 4747)])
@pytest.mark.parametrize("dtype,silu", [("float32", True), ("bfloat16", False)])
def test_long_runs_give_the_bits_of_small_steps(H, G, d, dv, rank, taps, total, dtype, silu, monkeypatch):
    from swifttransformer_b200 import ops
    monkeypatch.setattr(ops, "DELTA_CHUNK_MIN_TOKENS", 1 << 30)
    rng = np.random.default_rng(total)
    C = 2 * G * d + H * dv
    cols = C + H + (2 * rank if rank else H + H * dv)
    lens = []
    while sum(lens) < total - 120:
        lens.append([37, 100, 5, 61, 90, 13, 1, 2][len(lens) % 8])
    lens.append(total - sum(lens))
    proj = dev(rng.normal(size=(total, cols)))
    conv = dev(rng.normal(size=(C, taps)) * 0.5)
    low = lambda *s: dev(rng.normal(size=s) * 0.3, TD[dtype]) if rank else None
    a2, g2 = low(H * d, rank), low(H * dv, rank)
    a_log, norm = dev(rng.normal(size=H)), dev(1 + 0.1 * rng.normal(size=dv))
    dt_bias = dev(rng.normal(size=H * d if rank else H))
    tails0 = dev(rng.normal(size=(len(lens) + 1, taps - 1, C)))

    def run(rows, which, pad):
        st = Step([(i, 0, lens[i]) for i in which], pad_tokens=pad, pad_requests=0)
        rows = torch.cat([rows, torch.full((pad, cols), 7.0, device="cuda")])
        state = torch.zeros((len(lens) + 1, H, d, dv), device="cuda")
        scratch = torch.full((ops.delta_rule_scratch(st.n_rows, H, G, d, dv),), float("nan"), device="cuda")
        out = torch.full((st.n_rows, H * dv), 77.0, dtype=TD[dtype], device="cuda")
        ops.delta_rule(rows, C, C + H, C + H + (rank or H), conv, tails0.clone(), a2, a_log, dt_bias, g2, norm, 1e-5, 0.7, state, True,
                       False, scratch, out, st.positions, st.seq, st.q_start, st.slots, st.n_seqs, H, G, d, dv, gate_silu=silu)
        assert torch.all(out[st.n:] == 77.0)
        return out, state
    ops.delta_rule_set_lanes(8)
    try:
        out, state = run(proj, range(len(lens)), 7)
        at = 0
        for i, n in enumerate(lens):
            small, s = run(proj[at:at + n], [i], 1)
            assert torch.equal(small[:n], out[at:at + n]) and torch.equal(s[i], state[i]), i
            at += n
    finally:
        ops.delta_rule_set_lanes(0)
