"""The tcgen05 latent attention where a block has several query tiles one after the other, against float64."""
import math

import pytest
import torch

from test_latent_attention_tc_gpu import problem, run

pytestmark = pytest.mark.gpu


# 16 heads and two parts of the values (kr 512, 320): 74 blocks a part; tiles with one key tile to sixteen, and with as many as
# fit the window; the instance of known blocks and the general one, and one without blocks that are only keys
@pytest.mark.parametrize("H,kr,rot", [(16, 512, 64), (16, 320, 64), (12, 512, 0), (16, 256, 0)])
@pytest.mark.parametrize("runs,window", [([(0, 1000), (130, 700)], 0), ([(0, 1000), (130, 700)], 300), ([(5, 30), (0, 1400), (900, 9), (64, 300)], 70)])
def test_query_tiles_one_after_the_other(H, kr, rot, runs, window):
    ps = 16
    q, pool, gates, sink, rows, step = problem(runs, H, kr, rot, ps, H + window, window, pad=5)
    out, status = run(q, pool, gates, sink, step, H, kr, rot, ps, window)
    assert status == 0 and torch.all(out[q.shape[0] - 5:] == 77.0)
    at = 0
    for i, ((start, n), r) in enumerate(zip(runs, rows)):
        r = r.double()
        for h in range(H):                               # (the bounds of the short portions' test)
            x = (q[at:at + n].view(n, H, kr + rot)[:, h].double() @ r.T) * (kr / 4 + rot) ** -0.5
            p, j = torch.arange(start, start + n, device="cuda")[:, None], torch.arange(start + n, device="cuda")[None]
            x = x.masked_fill((j > p) | ((j <= p - window) if window else (j < 0)), -torch.inf)
            w = torch.cat([x, sink[h].double().expand(n, 1)], -1).softmax(-1)[:, :-1]
            f = torch.sigmoid(gates[at:at + n, h].double())[:, None]
            ref = (w @ r[:, :kr])
            bound = 2.0 ** -7 * (w @ r[:, :kr].abs()) + 2.0 ** -8 * ref.abs() + 1e-5
            got = out[at:at + n].view(n, H, kr)[:, h].double()
            assert torch.all((got - ref * f).abs() <= bound * f), (i, h)
        at += n
    # a request's last tokens, alone in a step of a few tiles, have the bits they have here (portions that begin with a tile)
    start, n = runs[1]
    first = sum(m for _, m in runs[:1])
    whole = 128 // math.gcd(128, H)
    a = (n - 40) // whole * whole
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    part = dict(step, positions=step["positions"][first + a:first + n].contiguous(), seq=ints([0] * (n - a)), q_start=ints([0, n - a, n - a]),
                start=ints([start + a, 0]), slots=ints([2, 0]), n_seqs=2)
    alone, status = run(q[first + a:first + n].contiguous(), pool, gates[first + a:first + n], sink, part, H, kr, rot, ps, window)
    assert status == 0 and torch.equal(alone, out[first + a:first + n])
