"""Every form of the 32-bit product (tiles of 8 and 16 rows on mma.sync, of 16 to 128 on tcgen05) gives the same bits."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


# outputs that fill tiles of 16 and 128 and that do not, several tiles a block; k in whole and ragged groups, fewer groups than warps, rows
# off 16 bytes
@pytest.mark.parametrize("k,outs,skip", [(768, 2304, 0), (132, 8200, 0), (2048, 130, 0), (70, 4000, 0), (100, 72, 1), (16, 9, 0), (8256, 24, 3)])
@pytest.mark.parametrize("rows", [1, 2, 7, 8, 9, 16, 23, 33, 64, 65, 140])
def test_forms(rows, k, outs, skip):
    from swifttransformer_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(k + outs + rows)
    cut = lambda n: torch.randn(n * k + skip, generator=gen, device="cuda")[skip:].view(n, k)
    a, w, bias = cut(rows), cut(outs), torch.randn(outs, generator=gen, device="cuda")
    chosen = ops.linear(a, w, bias, "relu")
    exact, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    bound = (k / 64 + 8) * 2.0 ** -23 * size + 2.0 ** -24 * (exact + bias).abs()          # (test_gemm_f32_parts_gpu.py) and the bias
    assert torch.all((chosen - torch.relu(exact + bias)).abs() <= bound)
    scratch = torch.empty(6 * rows * ((k + 63) // 64 * 64), dtype=torch.uint8, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    for form in [-8, -16] + list(range(16, 129, 16)):
        out = torch.full((rows + 1, outs), 77.0, device="cuda")
        assert ops.lib().st_gemm_f32(p(a), p(w), p(bias), p(out), rows, outs, k, ops.ACT_CODES["relu"], form, p(scratch), p(status),
                                     ops._stream()) == 0
        assert torch.equal(out[:rows], chosen) and torch.all(out[rows] == 77.0), form
    assert int(status) == 0
