"""The experts' products on tcgen05 at the edges of its tiles, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def order_of(counts, top, gen):
    """A step whose experts get these many items (the last -1 count: items no expert takes); -> (ops.ExpertOrder, tokens)."""
    from swifttransformer_b200 import ops
    e = torch.cat([torch.full((c,), i, dtype=torch.int32) for i, c in enumerate(counts)])
    drop = -len(e) % top
    e = torch.cat([e, torch.full((drop,), -1, dtype=torch.int32)])
    e = e[torch.randperm(len(e), generator=gen)].view(-1, top).cuda().contiguous()
    return ops.moe_sort(e, len(counts)), e.shape[0]


# counts: experts without items, one row, 31 to 33 (boxes of 32 rows), 127 to 129 and 256 / 257 (tiles of 128 rows)
COUNTS = [[1], [0, 3, 0, 0, 1], [33, 0, 127, 128, 129, 31, 32], [256, 5, 257, 1]]


@pytest.mark.parametrize("tile", [0, 64, 128, 256])
@pytest.mark.parametrize("gather,gated,act,k,n_out", [
    (True, True, "silu", 200, 200), (True, False, "none", 64, 296), (False, False, "gelu", 456, 33), (True, True, "relu2", 8, 72),
    (False, True, "silu", 1032, 136), (False, False, "none", 136, 520), (True, False, "silu", 2048, 31)])
@pytest.mark.parametrize("counts", COUNTS)
def test_products_in_every_tile(tile, gather, gated, act, k, n_out, counts, monkeypatch):
    from swifttransformer_b200 import ops
    monkeypatch.setattr(ops, "EXPERTS_TILE", tile)
    gen = torch.Generator().manual_seed(k + n_out)
    order, tokens = order_of(counts, 2, gen)
    rows = tokens if gather else order.n_items
    a = torch.randn((rows, k), generator=gen).to(torch.bfloat16).cuda()
    w = (torch.randn((len(counts), 2 * n_out if gated else n_out, k), generator=gen) * k ** -0.5).to(torch.bfloat16).cuda()
    got = ops.gemm_experts(a, w, order, gather, gated, act).double()
    assert ops.kernel_status(a.device) == 0
    f = {"none": lambda x: x, "silu": lambda x: x * torch.sigmoid(x), "relu2": lambda x: x.clamp(min=0) ** 2,
         "gelu": lambda x: 0.5 * x * (1 + torch.erf(x * 2 ** -0.5))}[act]
    offsets = order.offsets.tolist()
    for e, (lo, hi) in enumerate(zip(offsets, offsets[1:])):
        src = a[order.sorted[lo:hi].long() // 2] if gather else a[lo:hi]
        z = src.double() @ w[e].double().T
        sums = k * 2.0 ** -24 * (src.abs().double() @ w[e].abs().double().T)      # float sums in any order
        if gated:
            g, u = z[:, :n_out], z[:, n_out:]
            # either product may round to the neighbouring bfloat16: 2^-8 of itself, through act (|act'| <= 1.1, relu2 2 |g|)
            slope = 2 * g.abs() + 0.1 if act == "relu2" else torch.full_like(g, 1.1)
            bound = (2.0 ** -8 * g.abs() + sums[:, :n_out]) * slope * u.abs() * 1.1 \
                + f(g).abs() * (2.0 ** -8 * u.abs() + sums[:, n_out:]) * 1.1
            z = f(g) * u
        else:
            bound, z = sums * 1.2, f(z)
        bound = bound + 2.0 ** -8 * z.abs() + 1e-6            # the result's own rounding; the float functions
        assert torch.all((got[lo:hi] - z).abs() <= bound), (e, float(((got[lo:hi] - z).abs() - bound).max()))


@pytest.mark.parametrize("tile", [0, 64, 128, 256])
@pytest.mark.parametrize("clamp", [(7.0, 1.0, 1.0), (0.5, 1.702, 0.0), (1e30, 3.0, -1.0), (-1.0, 1.0, 1.0)])
@pytest.mark.parametrize("k,n_out,counts", [(200, 200, [33, 0, 129]), (1032, 31, [1]), (64, 136, [256, 5, 2])])
def test_the_clamped_unit_in_the_epilogue(tile, clamp, k, n_out, counts, monkeypatch):
    """The unit over the product's rows as they are stored, up to a neighbouring quotient: one bfloat16 of the result."""
    from swifttransformer_b200 import ops
    monkeypatch.setattr(ops, "EXPERTS_TILE", tile)
    gen = torch.Generator().manual_seed(k + n_out)
    order, tokens = order_of(counts, 2, gen)
    a = torch.randn((tokens, k), generator=gen).to(torch.bfloat16).cuda()
    w = (torch.randn((len(counts), 2 * n_out, k), generator=gen) * 4 * k ** -0.5).to(torch.bfloat16).cuda()
    a[0, 0], a[-1, 1] = float("inf"), float("nan")
    got = ops.gemm_experts(a, w, order, True, gated=True, clamp=clamp)
    want = ops.gated_clamped_act(ops.gemm_experts(a, w, order, True), None, *clamp)
    live = int(order.offsets[-1])
    got, want = got[:live].float(), want[:live].float()
    assert torch.equal(got.isnan(), want.isnan())
    same = (got == want) | want.isnan()
    assert torch.all(same | ((got - want).abs() <= 2.0 ** -7 * want.abs())) and same.float().mean() > 0.999
    assert ops.kernel_status(a.device) == 0


def test_a_row_does_not_depend_on_its_tile():
    from swifttransformer_b200 import ops
    gen = torch.Generator().manual_seed(1)
    a, w = torch.randn((300, 520), generator=gen).to(torch.bfloat16).cuda(), torch.randn((1, 264, 520), generator=gen).to(torch.bfloat16).cuda()
    whole = ops.gemm_experts(a, w, order_of([300], 1, gen)[0], gather=False)
    for n in (1, 32, 129):
        assert torch.equal(ops.gemm_experts(a[:n].contiguous(), w, order_of([n], 1, gen)[0], gather=False), whole[:n])


def test_silu_of_every_number(monkeypatch):
    """Through an identity: all finite bfloat16 numbers, and rows of the tile that no expert has beside them."""
    from swifttransformer_b200 import ops
    monkeypatch.setattr(ops, "EXPERTS_TILE", 64)
    a = torch.arange(1 << 16, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    a = a[torch.isfinite(a)].view(-1, 8).cuda()
    order, _ = order_of([len(a)], 1, torch.Generator().manual_seed(0))
    got = ops.gemm_experts(a, torch.eye(8, dtype=torch.bfloat16, device="cuda")[None].contiguous(), order, gather=False, act="silu")
    x = a.float()
    want = (x.double() / (1 + torch.exp(-x.double()))).to(torch.bfloat16)
    # float arithmetic, then the rounding: at most the neighbouring bfloat16 number; below -88.7, where exp(-x) leaves the floats,
    # zero for numbers up to 88.8 exp(-88.7) < 3e-37
    step = torch.maximum(want.double().abs() * 2.0 ** -7, torch.tensor(3e-37, dtype=torch.float64, device="cuda"))
    assert torch.all((got.double() - want.double()).abs() <= step)
    for bad, result in ((float("inf"), float("inf")), (float("nan"), float("nan"))):
        b = torch.zeros((3, 8), dtype=torch.bfloat16, device="cuda")
        b[1] = bad
        w = torch.ones((1, 8, 8), dtype=torch.bfloat16, device="cuda")
        out = ops.gemm_experts(b, w, order_of([3], 1, torch.Generator().manual_seed(0))[0], gather=False, act="silu")
        assert torch.all(out[::2] == 0) and torch.allclose(out[1].float(), torch.full((8,), result, device="cuda"), equal_nan=True)


def test_small_products_take_the_other_kernel():
    from swifttransformer_b200 import ops
    assert ops._experts_mma(8, 8, 256, 256) and not ops._experts_mma(8, 8, 264, 256) and not ops._experts_mma(512, 8, 256, 256)
