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
    for form in [0, -8, -16] + list(range(16, 129, 16)):
        out = torch.full((rows + 1, outs), 77.0, device="cuda")
        assert ops.lib().st_gemm_f32(p(a), p(w), p(bias), p(out), rows, outs, k, ops.ACT_CODES["relu"], form, p(scratch),
                                     ctypes.c_longlong(scratch.numel()), p(status), ops._stream()) == 0
        assert torch.equal(out[:rows], chosen) and torch.all(out[rows] == 77.0), form
    assert int(status) == 0


@pytest.mark.parametrize("rows,k,outs", [(700, 520, 2000), (257, 1032, 640), (129, 64, 20000), (20, 2048, 8192)])
def test_rows_in_parts(rows, k, outs, monkeypatch):
    """Scratch for some of the rows at a time: the same bits, and no more scratch than is allowed (a tile of 128 rows at least)."""
    from swifttransformer_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(rows)
    a, w, bias = (torch.randn(s, generator=gen, device="cuda") for s in ((rows, k), (outs, k), (outs,)))
    whole = ops.linear(a, w, bias, "gelu")
    per_row = 6 * ((k + 63) // 64 * 64)
    for most in (0, 300 * per_row, 10 ** 9):
        monkeypatch.setattr(ops, "GEMM_F32_SCRATCH", most)
        form, need = ops._gemm_f32_plan(rows, outs, k, most, a.device.index)
        assert form >= 16 and need == per_row * min(rows, max(most // (128 * per_row), 1) * 128)
        assert torch.equal(ops.linear(a, w, bias, "gelu"), whole)
    scratch, status = torch.empty(5 * per_row, dtype=torch.uint8, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    out, p = torch.empty_like(whole), lambda t: ctypes.c_void_p(t.data_ptr())
    for size, taken in ((5 * per_row, True), (per_row - 1, False)):  # (five rows at a time; not one)
        out.zero_()
        got = ops.lib().st_gemm_f32(p(a), p(w), p(bias), p(out), rows, outs, k, ops.ACT_CODES["gelu"], 16, p(scratch), ctypes.c_longlong(size),
                                    p(status), ops._stream())
        assert (got == 0) == taken and torch.equal(out, whole if taken else torch.zeros_like(whole))
    assert int(status) == 0
