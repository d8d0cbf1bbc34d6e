"""The 32-bit attention over tiles of query rows and over single tokens: the same bits as its general kernel (a block per
token and head), which queries that do not start on 16 bytes still go to."""
import random

import pytest
import torch

pytestmark = pytest.mark.gpu


def step(runs, page_size, heads, kv_heads, dim, layers, seed, pad):
    """runs: (slot, first position, tokens).  Keys and values past a request's last token are NaN, its last token's values
    infinite: neither may reach a row that does not see them."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n_slots = 1 + max(s for s, _, _ in runs)
    ends = [0] * n_slots
    for s, p, n in runs:
        ends[s] = max(ends[s], p + n)
    need = [-(-e // page_size) for e in ends]
    order = list(range(sum(need) + 1))
    random.Random(seed).shuffle(order)
    table = torch.full((n_slots, max(need) + 1), -1, dtype=torch.int32)
    pool = torch.full((len(order), layers, 2, kv_heads, page_size, dim), float("nan"), device="cuda")
    for s in range(n_slots):
        for j in range(need[s]):
            page = order.pop()
            table[s, j] = page
            live = min(page_size, ends[s] - j * page_size)
            pool[page, :, :, :, :live] = torch.randn((layers, 2, kv_heads, live, dim), generator=gen, device="cuda")
            if j == need[s] - 1:
                pool[page, :, 1, :, live - 1] = float("inf")
    pos = [p + i for _, p, n in runs for i in range(n)] + [-1] * pad
    seq = [k for k, (_, _, n) in enumerate(runs) for _ in range(n)] + [0] * pad
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    q = torch.randn((len(pos), heads * dim), generator=gen, device="cuda")
    return q, pool, ints(pos), ints(seq), ints([s for s, _, _ in runs]), table.cuda()


def both(q, pool, layer, args, heads, window):
    from swifttransformer_b200 import ops
    out, ref = torch.full_like(q, 77.0), torch.full_like(q, 77.0)
    status = torch.zeros(2, dtype=torch.int32, device="cuda")
    scale = pool.shape[-1] ** -0.5
    ops.attention_plain(q, pool, layer, out, *args, heads, scale, window, status[:1])
    odd = torch.empty(q.numel() + 1, device="cuda")[1:].view_as(q)
    odd.copy_(q)
    assert odd.data_ptr() % 16
    ops.attention_plain(odd, pool, layer, ref, *args, heads, scale, window, status[1:])
    return out, ref, status.tolist()


# runs of one token, of a tile of 32 and its edges, several in a tile, starting and ending at the edges of 32 and 128 keys, and
# of a few tokens
RUNS = [[(0, 0, 1)], [(0, 0, 300)], [(0, 127, 1), (1, 128, 1), (2, 700, 1), (3, 0, 1)], [(1, 0, 31), (0, 0, 33), (2, 95, 64)],
        [(0, 100, 2), (1, 0, 1), (2, 126, 5), (3, 255, 30), (4, 31, 1)], [(i, 3 * i, 1) for i in range(70)], [(0, 380, 129)],
        [(0, 120, 8), (1, 124, 9), (2, 0, 8), (3, 0, 9), (4, 500, 10), (5, 0, 3)]]


# (few heads: a block per token and head; with 256 of them most steps go by tiles of 32 rows)
@pytest.mark.parametrize("heads,kv_heads,dim,page_size", [(2, 2, 64, 16), (4, 2, 128, 8), (3, 3, 80, 7), (2, 1, 4, 16), (1, 1, 256, 32),
                                                          (2, 2, 132, 1), (1, 1, 20, 16), (256, 2, 64, 16), (256, 2, 128, 8),
                                                          (256, 1, 132, 7), (256, 1, 256, 32)])
@pytest.mark.parametrize("window", [0, 50, 128, 400])
def test_same_bits_as_the_general_kernel(heads, kv_heads, dim, page_size, window):
    for k, runs in enumerate(RUNS):
        q, pool, *args = step(runs, page_size, heads, kv_heads, dim, 2, k, pad=k % 3)
        out, ref, status = both(q, pool, 1, args, heads, window)
        assert status == [0, 0] and torch.equal(torch.nan_to_num(out, nan=5.0), torch.nan_to_num(ref, nan=5.0)), runs
        last = torch.tensor([p + n - 1 for _, p, n in runs], device="cuda", dtype=torch.int32)[args[1].long()]
        unseen = (args[0] >= 0) & (args[0] < last)
        assert torch.isfinite(out[unseen]).all() and torch.all(out[args[0] < 0] == 77.0)


def test_a_hole_in_the_block_table_is_reported():
    q, pool, pos, seq, slots, table = step([(0, 0, 200), (1, 300, 1)], 16, 2, 2, 64, 1, 3, 0)
    table[0, 3] = table[1, 2] = -1
    out, ref, status = both(torch.nan_to_num(q), torch.nan_to_num(pool, posinf=1.0), 0, (pos, seq, slots, table), 2, 0)
    assert status == [1, 1] and torch.equal(out, ref)
