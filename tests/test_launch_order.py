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
