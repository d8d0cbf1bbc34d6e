"""The 32-bit matrix product at the edges of its tiles, against float64 and against its general kernel bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# (rows, k, outputs): every tile of the dispatch with full and ragged edges in rows, outputs and k (k % 64, k < a stage)
SHAPES = [(1, 4, 1), (1, 2048, 2048), (4, 100, 2500), (5, 68, 33), (8, 2048, 7200), (8, 132, 4090), (8, 260, 700), (9, 64, 7130),
          (16, 516, 9000), (16, 36, 130), (17, 2048, 2117), (32, 1000, 4100), (33, 28, 65), (64, 8192, 129), (128, 300, 4500),
          (250, 96, 2050), (300, 768, 2304), (601, 340, 2047), (1000, 128, 2051), (2049, 44, 1283)]


@pytest.mark.parametrize("rows,k,outs", SHAPES)
def test_product_in_every_tile(rows, k, outs):
    from swifttransformer_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(rows * 7 + k)
    # (each operand inside a larger buffer whose margins are NaN: a row read past its end would show)
    def operand(n):
        buf = torch.full((n + 2, k), float("nan"), device="cuda")
        buf[1:-1] = torch.randn((n, k), generator=gen, device="cuda")
        return buf[1:-1]
    a, w = operand(rows), operand(outs)
    bias = torch.randn(outs, generator=gen, device="cuda")
    got = ops.linear(a, w, bias, "relu")
    # a chain of k fused multiply-adds and one sum: at most (k + 1) half-ulps of the running sums' bound |a| |w|
    bound = (k + 2) * 2.0 ** -24 * (a.abs().double() @ w.abs().double().T + bias.abs())
    exact = (a.double() @ w.double().T + bias.double()).clamp(min=0)
    assert torch.all((got.double() - exact).abs() <= bound)
    # rows that do not start on 16 bytes go to the general kernel: the same chain, the same bits
    odd = torch.empty(rows * k + 1, device="cuda")[1:].view(rows, k)
    odd.copy_(a)
    assert odd.data_ptr() % 16 and torch.equal(ops.linear(odd, w, bias, "relu"), got)


def test_a_row_does_not_depend_on_its_batch():
    from swifttransformer_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(3)
    a, w = torch.randn((700, 516), generator=gen, device="cuda"), torch.randn((2310, 516), generator=gen, device="cuda")
    whole = ops.linear(a, w)
    for n in (1, 3, 8, 11, 16, 29, 64, 200):
        assert torch.equal(ops.linear(a[:n], w), whole[:n]), n
