"""The 32-bit matrix product over few k: chains of multiply-adds, whose error the tensor cores' sums would exceed."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 2, 3, 4, 7, 8, 9, 15, 16])
@pytest.mark.parametrize("outs", [1, 64, 130])
def test_short_products(k, outs):
    from swifttransformer_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(k * outs)
    a, w = torch.randn((200, k), generator=gen, device="cuda"), torch.randn((outs, k), generator=gen, device="cuda")
    whole = ops.linear(a, w)
    if k <= 8:      # one rounding to nearest for each k, in ascending order (of a product that is exact in 64 bits)
        chain = torch.zeros_like(whole)
        for i in range(k):
            chain = (chain.double() + a[:, i:i + 1].double() * w[:, i].double()).float()
        assert torch.equal(whole, chain)
    for n in (1, 7, 8, 9, 33, 64, 65, 199):
        assert torch.equal(ops.linear(a[:n].contiguous(), w), whole[:n]) and torch.equal(ops.linear(a[200 - n:].contiguous(), w), whole[200 - n:])
    bias = torch.randn(outs, generator=gen, device="cuda")
    assert torch.equal(ops.linear(a, w, bias, "relu"), torch.relu(whole + bias))
