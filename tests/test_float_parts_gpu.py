"""Products of floats in three bfloat16 parts at the ends of the floats: numbers whose last part would fall under the smallest bfloat16, were
it not scaled up, and numbers whose first part is infinite for that."""
import numpy as np
import pytest
import torch

import test_delta_chunks_gpu as delta
import test_hgrn2_chunks_gpu as hgrn2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("e", [-100, -110, -114, -118, -122, -126, -130, -140])
@pytest.mark.parametrize("rows", [3, 8, 20, 40, 150])
def test_small_operands_of_a_product(rows, e):
    """Rows, or weights, of about 2^e against weights of 2^100: as close to 64 bits as ordinary ones (test_gemm_f32_parts_gpu.py has the bound),
    for each operand is taken as the float it is, down to those that are not normal."""
    from swifttransformer_b200 import ops
    k, outs = 520, 300
    gen = torch.Generator(device="cuda").manual_seed(rows - e)
    small, large = lambda n: torch.randn((n, k), generator=gen, device="cuda") * 2.0 ** e, lambda n: torch.randn((n, k), generator=gen, device="cuda") * 2.0 ** 100
    for a, w in ((small(rows), large(outs)), (large(rows), small(outs))):
        got, exact = ops.linear(a, w).double(), a.double() @ w.double().T
        bound = (k / 64 + 8) * 2.0 ** -23 * (a.abs().double() @ w.abs().double().T) + k * 2.0 ** -149
        assert torch.all((got - exact).abs() <= bound), float(((got - exact).abs() / bound).max())
        assert (got - exact).norm() <= 1.5e-7 * exact.norm()          # and, over all, the error of ordinary numbers: 1e-7


@pytest.mark.parametrize("e", [90, 96, 108, 112, 120, 125])
@pytest.mark.parametrize("rows", [3, 20, 150])
def test_large_operands_and_outputs_of_a_product(rows, e):
    """Rows of about 2^e with weights of 2^-90 (operands beyond 2^112) and of 1 (outputs beyond 2^96, and beyond the floats)."""
    from swifttransformer_b200 import ops
    k, outs = 200, 300
    gen = torch.Generator(device="cuda").manual_seed(rows + e)
    a, w = torch.randn((rows, k), generator=gen, device="cuda") * 2.0 ** e, torch.randn((outs, k), generator=gen, device="cuda")
    for w in (w * 2.0 ** -90, w):
        got, exact, size = ops.linear(a, w).double(), a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
        fits = size < 3e38                                # (a chain of k roundings at the most)
        assert torch.all(((got - exact).abs() <= k * 2.0 ** -24 * size)[fits])
        assert torch.all(got[exact.abs() > 3.5e38].isinf())
    assert ops.kernel_status(a.device) == 0


@pytest.mark.parametrize("e", [-112, -118, -122])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_small_values_of_the_hgrn2_recurrence(e, dtype, monkeypatch):
    H, d, dv, T = 2, 128, 64, 200
    p, f_bias, lower, norm_w = hgrn2.projections(T, H, d, dv, 5, "slow")
    p[:, 2 * H * d:] *= 2.0 ** e
    outs, states = [], []
    for chunks in (True, False):
        state = torch.zeros((2, H, d, dv), device="cuda")
        outs.append(hgrn2.scan([p], [T], [0], H, d, dv, f_bias, lower, norm_w, state, dtype, chunks, monkeypatch, [1])[0])
        states.append(state[1].double())
    assert (states[0] - states[1]).abs().max() <= 4e-6 * states[1].abs().max()          # (the bound of ordinary numbers)
    # float32 rows: as states; bfloat16 rows: two roundings to 8 bits
    assert np.abs(outs[0] - outs[1]).max() <= (4e-6 if dtype == "float32" else 2.0 ** -7) * np.abs(outs[1]).max()


@pytest.mark.parametrize("e", [-112, -118, -122])
def test_small_values_of_the_delta_rule(e, monkeypatch):
    H, G, d, dv, T = 2, 1, 128, 64, 200
    proj, w = delta.inputs(T, H, G, d, dv, 0, 7, "slow")
    proj[:, 2 * G * d:2 * G * d + H * dv] *= 2.0 ** e
    outs, states = [], []
    for chunks in (True, False):
        state, tails = torch.zeros((2, H, d, dv), device="cuda"), torch.zeros((2, 1, 2 * G * d + H * dv), device="cuda")
        outs.append(delta.step([proj], [T], [0], H, G, d, dv, 0, w, tails, state, "float32", chunks, monkeypatch, [1])[0])
        states.append(state[1].double())
    assert (states[0] - states[1]).abs().max() <= 4e-6 * states[1].abs().max()
    assert np.abs(outs[0] - outs[1]).max() <= 4e-6 * np.abs(outs[1]).max()
