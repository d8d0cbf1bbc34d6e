"""The HGRN2 recurrence in chunks where sums over a chunk are not finite, and with values next to the largest float."""
import numpy as np
import pytest
import torch

from test_hgrn2_chunks_gpu import projections, scan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,d,dv", [(2, 128, 128), (3, 64, 36), (1, 4, 8)])
@pytest.mark.parametrize("T,t0", [(65, 64), (128, 127), (150, 20), (150, 149)])
@pytest.mark.parametrize("dtype,value", [("float32", np.inf), ("float32", -np.inf), ("float32", np.nan), ("float32", 3.4e38), ("float32", -3.397e38),
                                         ("bfloat16", np.inf), ("bfloat16", 3.3e38)])
def test_a_value_out_of_range(H, d, dv, T, t0, dtype, value, monkeypatch):
    """An infinite value makes its column of the state infinite, a finite one above the largest bfloat16 number (in float32 rows) leaves it
    finite, the walk's numbers; the other columns and heads and the tokens before it keep theirs."""
    p, f_bias, lower, norm_w = projections(T, H, d, dv, T + d, "slow")
    lower = np.full_like(lower, 0.9)                  # (no product of gates underflows: infinity times zero is none)
    col = 2 * H * d + 3
    states, outs = {}, {}
    for chunks in (True, False):
        for x in (value, 1.0):
            q = p.copy()
            q[t0, col] = x
            state = torch.zeros((2, H, d, dv), device="cuda")
            outs[chunks, x] = scan([q], [T], [0], H, d, dv, f_bias, lower, norm_w, state, dtype, chunks, monkeypatch, [1])[0]
            states[chunks, x] = state[1].cpu().numpy()
    got, plain = states[True, value], states[True, 1.0]
    others = np.ones((H, d, dv), bool)
    others[0, :, 3] = False
    assert np.array_equal(got[others], plain[others])
    column = got[0, :, 3]
    if np.isfinite(value):                            # products of up to 150 gates and a few float roundings, in either order
        walk = states[False, value][0, :, 3]
        assert np.isfinite(column).all() and np.abs(column / 1e38 - walk / 1e38).max() <= 2e-5 * np.abs(walk / 1e38).max()
    else:
        assert np.isnan(column).all() if np.isnan(value) else (column == value).all()
        assert np.isnan(outs[True, value][t0:, 3]).all()
    assert np.array_equal(outs[True, value][:t0], outs[True, 1.0][:t0]) and np.array_equal(outs[True, value][:, dv:], outs[True, 1.0][:, dv:])
