"""The 32-bit matrix product of three bfloat16 parts per operand: one set of bits for every row count and kernel, and operands
whose sums are not finite."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# (k, outputs): groups of 64 k that are full, ragged and alone; one and several tiles of 16 and 128 outputs; both sides of the lines
# between the kernels (up to 8 rows, up to 32 by size, more)
@pytest.mark.parametrize("k,outs", [(64, 16), (2048, 2048), (768, 2304), (132, 8200), (4100, 130), (4160, 4112), (3, 40)])
def test_a_row_has_the_same_bits_in_every_batch(k, outs):
    from swifttransformer_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(k + outs)
    a, w = torch.randn((300, k), generator=gen, device="cuda"), torch.randn((outs, k), generator=gen, device="cuda")
    whole = ops.linear(a, w)
    exact = a.double() @ w.double().T
    # Each of the six products of a group of 64 k is cut off at 2^-23 of the running sum at most 4 times, of which only the last
    # four steps' sums are as large as the group's; then one rounding per group and the parts left out (2^-24): far
    # within k / 64 + 8 times 2^-23 of |a| |w|
    bound = (k / 64 + 8) * 2.0 ** -23 * (a.abs().double() @ w.abs().double().T)
    assert torch.all((whole.double() - exact).abs() <= bound)
    for n in (1, 8, 9, 16, 17, 24, 32, 33, 48, 64, 65, 100, 112, 128, 129):
        assert torch.equal(ops.linear(a[:n].contiguous(), w), whole[:n]), n
        assert torch.equal(ops.linear(a[300 - n:].contiguous(), w), whole[300 - n:]), n
    assert ops.kernel_status(a.device) == 0


@pytest.mark.parametrize("rows", [3, 12, 40, 150])
def test_operands_that_are_not_finite(rows):
    """Infinities, NaN, sums beyond the floats and operands next to the largest float give what a chain over k gives."""
    from swifttransformer_b200 import ops
    k, outs = 100, 200
    gen = torch.Generator().manual_seed(rows)
    a, w = torch.randn((rows, k), generator=gen), torch.randn((outs, k), generator=gen)
    a[0, 5], a[1, 99], a[2, 64] = float("inf"), float("nan"), 3.4e38
    w[7, 70], w[8, 2], w[199, 5] = float("-inf"), 3.4028e38, 0.0
    a[:, 70].abs_()
    for act in ("none", "relu", "gelu"):
        got = ops.linear(a.cuda(), w.cuda(), None, act).cpu().numpy()
        with np.errstate(all="ignore"):
            an, wn = a.numpy(), w.numpy()
            chain = np.zeros((rows, outs), np.float32)
            for i in range(k):               # (a rounding of the product more than a fused chain has: compared within a bound)
                chain = (chain.astype(np.float64) + an[:, i:i + 1].astype(np.float64) * wn[None, :, i].astype(np.float64)).astype(np.float32)
            if act == "relu":                # (the kernels' is v > 0 ? v : 0)
                want = np.where(chain > 0, chain, np.float32(0))
            elif act == "gelu":
                x = chain.astype(np.float64)
                want = (0.5 * x * (1 + torch.erf(torch.from_numpy(x * 0.5 ** 0.5)).numpy())).astype(np.float32)
            else:
                want = chain
        assert np.array_equal(np.isnan(got), np.isnan(want)), act
        inf = np.isinf(want)
        assert np.array_equal(got[inf], want[inf])
        ok = np.isfinite(want)
        scale = (np.abs(np.where(np.isfinite(an), an, 0)).astype(np.float64) @ np.abs(np.where(np.isfinite(wn), wn, 0)).T.astype(np.float64))
        assert np.all(np.abs(got[ok].astype(np.float64) - want[ok]) <= (k + 2) * 2.0 ** -23 * scale[ok] + 1e-30)
    assert ops.kernel_status(torch.device("cuda")) == 0


@pytest.mark.parametrize("rows,k,outs", [(300, 520, 8200), (1000, 16384, 4096), (64, 768, 21000), (21, 2050, 40000)])
@pytest.mark.parametrize("act", ["none", "relu", "gelu"])
def test_rows_that_are_not_finite_in_tiles_one_after_the_other(rows, k, outs, act):
    """Products whose outputs are for the most part not finite, several tiles a block: all of them are formed, no wait runs out, and the rows
    beside them have the bits they have alone."""
    from swifttransformer_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(rows)
    a, w = torch.randn((rows, k), generator=gen, device="cuda"), torch.randn((outs, k), generator=gen, device="cuda")
    bias = torch.randn(outs, generator=gen, device="cuda")
    clean = ops.linear(a, w, bias, act)
    bad = a.clone()
    bad[::3, k - 7] = float("inf")                       # infinite outputs, their sign that of the weight
    bad[1::3, 5] = float("nan")
    got = ops.linear(bad, w, bias, act)
    want = clean.clone()
    want[::3] = torch.where(w[:, k - 7] > 0, float("inf"), float("-inf"))
    want[1::3] = float("nan")
    if act == "relu":                                    # (the kernels' is v > 0 ? v : 0)
        want = torch.where(want > 0, want, 0.0)
    elif act == "gelu":                                  # -inf times zero
        want = torch.where(want == float("-inf"), float("nan"), want)
    assert torch.equal(got.isnan(), want.isnan())
    assert torch.all((got == want) | want.isnan())
    assert ops.kernel_status(a.device) == 0
