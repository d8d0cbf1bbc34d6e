"""Sums over a chunk of the gated delta rule that are not finite: the categories of the walk token by token."""
import numpy as np
import pytest
import torch

from test_delta_chunks_gpu import inputs, step

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,d,dv", [(2, 64, 36), (40, 64, 36), (3, 100, 4)])      # eight and sixteen columns a block, ragged ones
@pytest.mark.parametrize("T", [65, 128, 150])
@pytest.mark.parametrize("value", [np.inf, 3.4e38])
def test_a_last_value_out_of_range(H, d, dv, T, value, monkeypatch):
    """An infinite value in the last token, or one above the largest bfloat16 number: its column of the state has the walk's infinities,
    signs included, and the other columns and heads their numbers."""
    proj, w = inputs(T, H, 1, d, dv, 0, T + d, "slow")
    C, col = 2 * d + H * dv, 2 * d + 3
    w["conv"][col] = [0.0, 1.0]
    states = {}
    for chunks in (True, False):
        for x in (value, 1.0):
            p = proj.copy()
            p[T - 1, col] = x
            state, tails = torch.zeros((2, H, d, dv), device="cuda"), torch.zeros((2, 1, C), device="cuda")
            step([p], [T], [0], H, 1, d, dv, 0, w, tails, state, "float32", chunks, monkeypatch, [1])
            states[chunks, x] = state[1].cpu().numpy()
    got, walk, plain = states[True, value], states[False, value], states[True, 1.0]
    others = np.ones((H, d, dv), bool)
    others[0, :, 3] = False
    assert np.array_equal(got[others], plain[others])
    assert np.array_equal(np.isnan(got), np.isnan(walk)) and np.array_equal(np.isinf(got), np.isinf(walk))
    assert np.array_equal(np.sign(got[np.isinf(got)]), np.sign(walk[np.isinf(walk)]))
    if np.isinf(value):
        assert np.isinf(got[0, :, 3]).any()
    else:                                             # sums of a few float roundings, in either order
        assert np.abs(got[0, :, 3] / 1e38 - walk[0, :, 3] / 1e38).max() <= 1e-5 * np.abs(walk[0, :, 3] / 1e38).max()
