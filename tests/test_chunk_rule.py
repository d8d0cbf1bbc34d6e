"""Which requests of a step run in chunks, and where their chunks stand: the arithmetic of csrc/chunks.cuh, on the CPU."""
import random

import pytest

from swifttransformer_b200 import ops

C = 64


def place(begin, b, start):
    return begin // C + min(b, begin // start)


@pytest.mark.parametrize("start", [1, 2, 63, 64, 65, 96, 112, 168, 256, 288])
def test_chunks_stand_apart_and_are_found(start):
    rng = random.Random(start)
    for _ in range(300):
        lens = [rng.choice([0, 1, 1, 2, start - 1, start, start + 1, C - 1, C, C + 1, rng.randrange(0, 700)])
                for _ in range(rng.randrange(1, 12))]
        q = [0]
        for n in lens:
            q.append(q[-1] + n)
        total = q[-1] + rng.choice([0, 1, 63, 127])              # padding tokens behind, and requests without tokens
        q += [q[-1]] * rng.randrange(0, 4)
        n_seqs = len(q) - 1
        stand = {}
        for b, n in enumerate(lens):
            if n >= start:
                for c in range(-(-n // C)):
                    p = place(q[b], b, start) + c
                    assert p not in stand
                    stand[p] = (b, c)
        longs = min(n_seqs, total // start) if total >= start else 0
        places = -(-total // C) + longs - 1 if longs else 0
        assert len(stand) == 0 or max(stand) < places
        for p in range(places):
            lo, hi = 0, n_seqs
            while hi - lo > 1:
                mid = (lo + hi) // 2
                lo, hi = (mid, hi) if place(q[mid], mid, start) <= p else (lo, mid)
            c, n = p - place(q[lo], lo, start), q[lo + 1] - q[lo]
            found = (lo, c) if c >= 0 and n - c * C > 0 and n >= start else None
            assert found == stand.get(p)


def test_the_rule():
    # portions, line -> (requests of so many tokens and more in chunks, what else walks: nothing, few tokens each, portions)
    for lens, limit, want in (([95, 1], 96, (0, 1)), ([96], 96, (96, 0)), ([2000, 96], 96, (96, 0)), ([2000, 1, 1, 3], 96, (96, 1)),
                              ([2000, 60, 1], 96, (96, 2)), ([], 96, (0, 1)), ([1] * 300, 96, (0, 1))):
        assert ops.chunk_split(lens, limit) == want
    # the line rises with the work of narrow heads, up to twice
    assert [ops._hgrn2_chunks_from(n, 16, 16, 64) for n in (300, 1600, 2000, 8000)] == [96, 142, 168, 192]
    assert ops._hgrn2_chunks_from(8000, 16, 16, 128) == 96 and ops._hgrn2_chunks_from(8000, 1, 16, 64) == 112
    assert ops._hgrn2_chunks_from(128, 1, 8, 64) == 144 and ops._hgrn2_chunks_from(128, 1, 4, 128) == 112
    assert ops.delta_split([287], 320, 1) == (0, 1) and ops.delta_split([288], 320, 1) == (288, 0)
    assert ops.delta_split([256, 1], 320, 2) == (256, 1)
    # the step's shape alone: all or none
    assert ops._split_of(191, 2, 96) == (0, 1) and ops._split_of(192, 2, 96) == (1, 0)


def test_scratch_holds_every_request_in_chunks():
    for lens, n, seqs in (([2000], 2000, 1), ([2000] + [1] * 32, 2048, 48), ([100] * 4, 448, 4), ([128], 128, 1), ([95, 2], 128, 2),
                          ([96] * 21, 2016, 24)):
        for H, d, vd in ((16, 128, 128), (4, 64, 128), (2, 20, 40)):
            split = ops.hgrn2_split(lens, n, seqs, H, d)
            need = (-(-n // C) + min(seqs, n // split[0]) - 1) * H * d * (vd + 1) if split[0] else 0
            assert ops.hgrn2_scratch(n, seqs, H, d, vd, split) == max(need, n * H * (vd + 2 * d))
            split = ops.delta_split(lens, n, seqs)
            need = int(ops.lib().st_delta_rule_chunk_floats(n, min(seqs, n // split[0]), H, H, d, vd)) if split[0] else 0
            assert ops.delta_rule_scratch(n, H, H, d, vd, seqs, split) == max(
                need, int(ops.lib().st_delta_rule_scratch_floats(n, H, H, d, vd)))
            assert ops.delta_rule_scratch(n, H, H, d, vd) >= ops.delta_rule_scratch(n, H, H, d, vd, seqs, split)
