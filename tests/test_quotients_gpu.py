"""The sigmoid and SiLU of the recurrences, the experts' units and the norm of the chunked recurrence against 64 bits over the whole range:
borders of the exponential, results that are not normal, infinities and numbers that are none."""
import numpy as np
import pytest
import torch

from test_fanidra_gpu import Step, dev
from test_gemm_experts_gpu import order_of

pytestmark = pytest.mark.gpu

FLT_MAX = 3.4028234663852886e38


@pytest.mark.parametrize("n", [100, 160])                # the preparation of small steps, and by runs of tokens
def test_sigmoid_and_silu(n):
    """As ``delta_rule`` leaves them in its scratch: SiLU of the values, sigmoid of the write strengths."""
    from swifttransformer_b200 import ops
    rng = np.random.default_rng(0)
    H = G = 4
    d = dv = 32
    z = np.concatenate([rng.uniform(-110, 110, 1500), rng.normal(size=1500), np.linspace(-89, -86, 400), np.linspace(86, 89, 100),
                        [0.0, -0.0, 1e-30, -1e-30, 1e-45, FLT_MAX, -FLT_MAX, -103.9, -104.0, np.inf, -np.inf, np.nan, 16.6, -16.6]])
    z = np.concatenate([z, np.zeros(-len(z) % (n * H))]).astype(np.float32)
    C = 2 * G * d + H * dv
    for part in z.reshape(-1, n, H):
        proj = np.zeros((n, C + H + H + H * dv), np.float32)
        proj[:, 2 * G * d:C] = np.repeat(part, dv, axis=1)
        proj[:, C:C + H] = part
        st = Step([(i, 0, 1) for i in range(n)])          # requests of a token each: a number meets no other one in the convolution
        conv = torch.zeros((C, 2), device="cuda")
        conv[:, 1] = 1.0
        scratch = torch.full((ops.delta_rule_scratch(n, H, G, d, dv),), 5.0, device="cuda")
        ops.delta_rule(dev(proj), C, C + H, C + 2 * H, conv, torch.zeros((n, 1, C), device="cuda"), None, torch.zeros(H, device="cuda"),
                       torch.zeros(H, device="cuda"), None, torch.ones(dv, device="cuda"), 1e-5, 1.0, torch.zeros((n, H, d, dv), device="cuda"),
                       False, False, scratch, torch.empty((n, H * dv), device="cuda"), st.positions, st.seq, st.q_start, st.slots, n, H, G, d, dv)
        stride = C + H * d + H
        rows = scratch[:n * stride].view(n, stride).cpu().numpy()
        with np.errstate(all="ignore"):
            e = np.exp(-part.astype(np.float64))
            den = 1.0 + np.where(e > FLT_MAX, np.inf, e)
            for got, want in ((rows[:, 2 * G * d:C].reshape(n, H, dv), (part / den)[:, :, None].repeat(dv, 2)), (rows[:, stride - H:], 1.0 / den)):
                assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isinf(got), np.isinf(want))
                ok = np.isfinite(want)
                # an exponential within 2 units of the last place, a sum, a quotient next to its last bit; where the result is not normal its step
                assert np.all(np.abs(got[ok] - want[ok]) <= 4 * 2.0 ** -23 * np.abs(want[ok]) + 2.0 ** -149)


@pytest.mark.parametrize("clamp", [None, (7.0, 1.702, 1.0), (1e30, 1.0, 0.0)])
def test_the_experts_units(clamp):
    """Every finite bfloat16 as a gate, against ups of all sizes: one rounding to bfloat16, beside the float's own."""
    from swifttransformer_b200 import ops
    gate = torch.arange(65536, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    gate = gate[gate.float().isfinite()]
    gen = torch.Generator().manual_seed(3)
    n, k, outs = len(gate), 16, 64
    order, tokens = order_of([n], 1, gen)
    assert tokens == n and not ops._experts_mma(order.n_items, 1, 2 * outs, k)
    a = torch.zeros((n, k), dtype=torch.bfloat16)
    a[:, 0], a[:, 1] = gate, (torch.randn(n, generator=gen) * 8).to(torch.bfloat16)
    w = torch.zeros((1, 2 * outs, k), dtype=torch.bfloat16)
    w[0, :outs, 0], w[0, outs:, 1] = 1, 1
    got = ops.gemm_experts(a.cuda(), w.cuda(), order, True, gated=True, act="silu", clamp=clamp).double().cpu()
    place = order.sorted.cpu().long()
    g, u = a[place, 0].double()[:, None], a[place, 1].double()[:, None]
    alpha, shift = 1.0, 0.0
    if clamp is not None:
        limit, alpha, shift = clamp
        g, u = g.clamp(max=limit), u.clamp(-limit, limit)
    e = torch.exp(-alpha * g)
    want = (g / (1 + torch.where(e > FLT_MAX, torch.inf, e)) * (u + shift)).expand(n, outs)
    big = want.abs() > 3.3895e38                          # (rounds beyond the largest bfloat16)
    assert torch.all(got[big].isinf() | (got[big].abs() > 3.38e38))
    off = ((got - want).abs() > (2.0 ** -8 + 2.0 ** -20) * want.abs() + 2.0 ** -134) & ~big
    assert not off.any(), [x[off][:6].tolist() for x in (got, want, g.expand(n, outs), u.expand(n, outs))]
    assert ops.kernel_status(torch.device("cuda")) == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_the_norm_of_the_chunked_recurrence(dtype, monkeypatch):
    """Gates that forget everything: a token's sum is a multiple of its own values, of any size."""
    from swifttransformer_b200 import ops
    monkeypatch.setattr(ops, "HGRN2_CHUNK_MIN_TOKENS", 1)
    H, d, dv, T = 2, 4, 32, 192
    rng = np.random.default_rng(1)
    v = torch.tensor(rng.normal(size=(T, H, dv)) * 2.0 ** rng.integers(-52, 52, size=(T, H, 1)), dtype=torch.float32).to(dtype)
    proj = torch.cat([torch.full((T, H * d), 20.0), torch.full((T, H * d), -300.0), v.float().view(T, -1)], 1).to(dtype).cuda()
    st = Step([(0, 0, T)])
    out, state = torch.empty((T, H * dv), dtype=dtype, device="cuda"), torch.zeros((1, H, d, dv), device="cuda")
    scratch = torch.zeros(max(int(ops.lib().st_hgrn2_chunks_scratch(T, 1, H, d, dv)), T * H * dv), device="cuda")
    zero = torch.zeros(H * d, device="cuda")
    ops.hgrn2_scan(proj, 0, H * d, 2 * H * d, zero, zero, torch.ones(dv, device="cuda"), 1e-33, state, out, st.positions, st.q_start, st.slots, 1,
                   H, d, dv, scratch=scratch, split=(1, 0))
    o = v.double() * (d * 20.0 / (1 + np.exp(-20.0)))
    want = o / ((o * o).mean(-1, keepdim=True) + 1e-33).sqrt()
    got = out.double().cpu().view(T, H, dv)
    # sums of 32 squares and of a few products in float, and the row's own rounding
    assert torch.all((got - want).abs() <= (4e-6 + (2.0 ** -8 if dtype == torch.bfloat16 else 0)) * want.abs())
