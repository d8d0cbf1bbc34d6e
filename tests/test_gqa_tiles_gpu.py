"""Grouped attention for prompt portions where its blocks of 64 or 128 query rows begin and end, against 64-bit arithmetic."""
import numpy as np
import pytest
from test_norelix_gpu import GqaCase

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("window,keep", [(0, 0), (65, 3)])
@pytest.mark.parametrize("d,vd", [(32, 32), (64, 128), (64, 136), (72, 128), (128, 64)])
def test_portions_that_end_at_the_blocks_edges(d, vd, window, keep):
    lengths = [16, 63, 64, 65, 127, 128, 129, 193, 257]
    case = GqaCase(lengths, 4, 2, d, vd, 16, seed=d + vd, dtype="bfloat16", window=window, keep_first=keep, sink=0.5, gate=False)
    case.write_pool()
    got = case.run([(i, 0, n) for i, n in enumerate(lengths)], "tiles")
    portion = case.run([(i, n // 3, n - n // 3) for i, n in enumerate(lengths)], "tiles")
    # a weight rounded to bfloat16 is off by at most 2^-9 of itself and the weights add up to at most one; the result's own
    # rounding is 2^-9 of it; the float scores and exponentials stay well below 1e-3
    for i, n in enumerate(lengths):
        tol = (2 * 2.0 ** -9 + 1e-3) * np.abs(case.v[i]).max()
        ref = case.reference(i)
        assert np.abs(got[i] - ref).max() <= tol
        # which rows share a block changes no number, so a portion's rows are the whole prompt's
        assert np.array_equal(portion[i], got[i][n // 3:])
