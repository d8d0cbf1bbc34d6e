"""The order in which kernels take tensor memory and let their successors in, read from the sources."""
import os
import re

import pytest

from swifttransformer_b200.ops import build


def bodies():
    """The text of every kernel that allocates tensor memory, up to the next kernel of its file."""
    for name in build.sources():
        with open(os.path.join(build.CSRC, name)) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for i, part in enumerate(text.split("__global__")[1:]):
            if "tcgen05.alloc." in part:
                yield pytest.param(part, id=f"{name}-{i}")


@pytest.mark.parametrize("body", list(bodies()))
def test_a_successor_comes_in_behind_the_allocation(body):
    """A successor's block may allocate before it waits for this grid; a grid that had triggered and then found too few
    columns would wait for the successor, and the successor for it."""
    trigger = body.find("ST_PDL_TRIGGER()")
    if trigger < 0:
        return
    barrier = body.find("__syncthreads()", body.rfind("tcgen05.alloc."))
    assert 0 <= barrier < trigger


@pytest.mark.gpu
def test_a_successor_that_allocates_first():
    """Latent attention of a row small enough to share a multiprocessor with the experts' product behind it."""
    import torch
    import test_latent_attention_tc_gpu as latent
    from swifttransformer_b200 import ops
    H, kr, rot, ps = 16, 64, 0, 16
    q, pool, gates, sink, _, step = latent.problem([(0, 700), (100, 500)], H, kr, rot, ps, 1)
    order = ops.moe_sort(torch.arange(600, dtype=torch.int32, device="cuda").view(300, 2) % 8, 8)
    a = torch.randn((300, 512), device="cuda").to(torch.bfloat16)
    w = (torch.randn((8, 1024, 512), device="cuda") * 0.05).to(torch.bfloat16)
    alone = latent.run(q, pool, gates, sink, step, H, kr, rot, ps, 0)[0], ops.gemm_experts(a, w, order, True, True, "silu")
    torch.cuda.synchronize()
    out, status = torch.empty_like(alone[0]), torch.zeros(1, dtype=torch.int32, device="cuda")
    for _ in range(50):
        ops.latent_attention(q, pool, 1, out, step["positions"], step["seq"], step["slots"], step["table"], H, kr, rot, ps,
                             (kr / 4 + rot) ** -0.5, sink, gates, status=status, kernel="tc", q_start=step["q_start"],
                             start_pos=step["start"], n_seqs=step["n_seqs"])
        y = ops.gemm_experts(a, w, order, True, True, "silu")
    assert torch.equal(out, alone[0]) and torch.equal(y, alone[1])
    assert int(status.item()) == 0 and ops.kernel_status(a.device) == 0
