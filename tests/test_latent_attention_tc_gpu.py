"""The tcgen05 latent attention against float64 at the edges of its tiles of 128 rows and 64 keys."""
import random

import pytest
import torch

pytestmark = pytest.mark.gpu


def problem(runs, H, kr, rot, ps, seed, window=0, pad=0):
    """runs: (start, tokens) per request.  Pages behind the window are taken out of the block table; spare pages and the rows
    that no query sees (past a request's last token, behind the window) are not numbers."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kd = kr + rot
    need = [-(-(s + n) // ps) for s, n in runs]
    order = list(range(sum(need) + 1))
    random.Random(seed).shuffle(order)
    table = torch.full((len(runs) + 1, max(need) + 1), -1, dtype=torch.int32)
    pool = torch.full((len(order), 2, ps, kd), float("nan"), dtype=torch.bfloat16, device="cuda")
    rows, k = [], 0
    for i, (s, n) in enumerate(runs):
        r = torch.randn((s + n, kd), generator=gen, device="cuda").to(torch.bfloat16)
        rows.append(r)
        for j in range(need[i]):
            page = order[k]
            k += 1
            if not window or (j + 1) * ps > s - window + 1:
                table[i + 1, j] = page
            part = r[j * ps:(j + 1) * ps]
            unseen = min(max(s - window + 1 - j * ps, 0), len(part)) if window else 0
            pool[page, 1, unseen:len(part)] = part[unseen:]
    n_all = sum(n for _, n in runs)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    q_start = [0]
    for _, n in runs:
        q_start.append(q_start[-1] + n)
    q = (torch.randn((n_all + pad, H * kd), generator=gen, device="cuda") * 0.7).to(torch.bfloat16)
    wide = torch.randn((n_all + pad, H + 3), generator=gen, device="cuda").to(torch.bfloat16)
    sink = torch.randn(H, generator=gen, device="cuda")
    pos = [s + j for s, n in runs for j in range(n)] + [-1] * pad
    seq = [i for i, (_, n) in enumerate(runs) for _ in range(n)] + [0] * pad
    step = dict(positions=ints(pos), seq=ints(seq), slots=ints(list(range(1, len(runs) + 1)) + [0]), table=table.cuda(),
                q_start=ints(q_start + [n_all]), start=ints([s for s, _ in runs] + [0]), n_seqs=len(runs) + 1)
    return q, pool.view(len(order), 2, ps * kd), wide[:, 2:2 + H], sink, rows, step


def run(q, pool, gates, sink, step, H, kr, rot, ps, window, kernel="tc"):
    from swifttransformer_b200 import ops
    out = torch.full((q.shape[0], H * kr), 77.0, dtype=torch.bfloat16, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    ops.latent_attention(q, pool, 1, out, step["positions"], step["seq"], step["slots"], step["table"], H, kr, rot, ps,
                         (kr / 4 + rot) ** -0.5, sink, gates, status=status, kernel=kernel, q_start=step["q_start"],
                         start_pos=step["start"], n_seqs=step["n_seqs"], window=window)
    return out, int(status.item())


RUNS = [[(0, 1)], [(0, 8)], [(0, 9)], [(63, 2), (0, 64), (130, 1)], [(0, 150), (57, 23)], [(200, 40), (0, 3), (64, 65)]]


@pytest.mark.parametrize("H,kr,rot,ps", [(16, 512, 64, 16), (5, 512, 0, 8), (8, 256, 64, 32), (3, 64, 0, 64), (16, 320, 64, 16),
                                         (1, 128, 128, 8), (4, 448, 128, 16), (128, 192, 0, 16)])
@pytest.mark.parametrize("window", [0, 40, 64])
def test_portions(H, kr, rot, ps, window):
    for k, runs in enumerate(RUNS):
        q, pool, gates, sink, rows, step = problem(runs, H, kr, rot, ps, 10 * k + H, window, pad=k % 3)
        g, s = (gates, sink) if k % 2 == 0 else (None, None)
        out, status = run(q, pool, g, s, step, H, kr, rot, ps, window)
        assert status == 0
        at = 0
        for (start, n), r in zip(runs, rows):
            r = r.double()
            x = (q[at:at + n].double().view(n, H, kr + rot).transpose(0, 1) @ r.T) * (kr / 4 + rot) ** -0.5
            p, j = torch.arange(start, start + n, device="cuda")[:, None], torch.arange(start + n, device="cuda")[None]
            x = x.masked_fill((j > p) | ((j <= p - window) if window else (j < 0)), -torch.inf)
            x = torch.cat([x, (s.double() if s is not None else torch.full((H,), -torch.inf, device="cuda").double())[:, None, None].expand(H, n, 1)], -1)
            w = x.softmax(-1)[..., :-1]
            ref = (w @ r[:, :kr]).transpose(0, 1)
            # weights rounded to bfloat16 (2^-9 each, and of their sum), the result's own rounding
            bound = 2.0 ** -7 * (w @ r[:, :kr].abs()).transpose(0, 1) + 2.0 ** -8 * ref.abs() + 1e-5
            if g is not None:
                f = torch.sigmoid(g[at:at + n].double())[:, :, None]
                ref, bound = ref * f, bound * f
            got = out[at:at + n].double().view(n, H, kr)
            assert torch.all((got - ref).abs() <= bound), (k, float(((got - ref).abs() / bound).max()))
            at += n
        assert torch.all(out[at:] == 77.0)


def test_a_row_does_not_depend_on_its_portion():
    q, pool, gates, sink, _, step = problem([(0, 300)], 16, 512, 64, 16, 3)
    whole, _ = run(q, pool, gates, sink, step, 16, 512, 64, 16, 0)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    for a, n in ((0, 8), (16, 40), (96, 204)):
        part = dict(step, positions=step["positions"][a:a + n].contiguous(), seq=step["seq"][a:a + n].contiguous(),
                    q_start=ints([0, n, n]), start=ints([a, 0]))
        out, status = run(q[a:a + n].contiguous(), pool, gates[a:a + n], sink, part, 16, 512, 64, 16, 0)
        assert status == 0 and torch.equal(out, whole[a:a + n])


def test_a_hole_in_the_block_table_is_reported():
    q, pool, gates, sink, _, step = problem([(0, 200)], 16, 512, 64, 16, 4)
    step["table"][1, 3] = -1
    out, status = run(q, pool, gates, sink, step, 16, 512, 64, 16, 0)
    assert status == 1 and torch.isfinite(out.float()).all()


def test_prompts_take_it_and_single_tokens_do_not(monkeypatch):
    """The rule of ``kernel="auto"``: what a step's shape is given to."""
    from swifttransformer_b200 import ops
    for runs, tc in (([(0, 600)], True), ([(100, 1)], False), ([(0, 20)], False)):
        q, pool, gates, sink, _, step = problem(runs, 16, 512, 64, 16, 5)
        auto, _ = run(q, pool, gates, sink, step, 16, 512, 64, 16, 0, "auto")
        want, _ = run(q, pool, gates, sink, step, 16, 512, 64, 16, 0, "tc" if tc else "mma")
        assert torch.equal(auto, want)


def test_a_result_off_sixteen_bytes_is_still_taken():
    from swifttransformer_b200 import ops
    H, kr, rot, ps, n = 16, 512, 64, 16, 600
    q, pool, gates, sink, _, step = problem([(0, n)], H, kr, rot, ps, 6)
    outs = []
    for kernel, skip in (("mma", 0), ("auto", 2)):
        outs.append(torch.full((n * H * kr + skip,), 77.0, dtype=torch.bfloat16, device="cuda")[skip:].view(n, H * kr))
        ops.latent_attention(q, pool, 1, outs[-1], step["positions"], step["seq"], step["slots"], step["table"], H, kr, rot, ps,
                             (kr / 4 + rot) ** -0.5, sink, gates, kernel=kernel, q_start=step["q_start"], start_pos=step["start"],
                             n_seqs=step["n_seqs"])
    assert torch.equal(*outs)
