"""The step plan of the recurrences that run long portions in chunks of tokens side by side."""
from __future__ import annotations

from typing import Any, Callable, Tuple

from .base import StepPlan


class PortionPlan(StepPlan):
    """Which requests of a step run in chunks and whether others walk (``ops.chunk_split``).  It holds no arrays: the kernels
    find the requests on the device, and a recorded step only agrees in what is launched."""

    def __init__(self, name: str, split: Callable[..., Tuple[int, int]]):
        self.name, self._split = name, split          # split(lens, tokens, requests of the step with its padding)

    def shape_key(self, lens, start, n_cap: int, b_cap: int) -> Tuple:
        return self._split(lens, n_cap, b_cap)

    def fill(self, lens, q_start, start, out, n_cap: int, b_cap: int) -> Tuple:
        return self._split(lens, n_cap, b_cap)

    def view(self, dev, key: Tuple, n_cap: int, b_cap: int) -> Any:
        return key
