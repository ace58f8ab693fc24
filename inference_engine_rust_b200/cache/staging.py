"""Page-locked host memory for what a step sends to the device: copies from it do not make the host wait for the device."""
from __future__ import annotations

from typing import List, Optional, Tuple

import torch


class PinnedRing:
    """Pinned host buffers for integers on their way to the device, used in rotation so that a buffer
    is rewritten only after its copy to the device has finished."""

    def __init__(self, depth: int = 4):
        self.depth = depth
        self.host: List[Optional[torch.Tensor]] = [None] * depth
        self.events: List[Optional[torch.cuda.Event]] = [None] * depth
        self.turn = 0

    def next(self, n_ints: int) -> Tuple[torch.Tensor, int]:
        i = self.turn
        self.turn = (self.turn + 1) % self.depth
        if self.events[i] is not None:
            self.events[i].synchronize()
        buf = self.host[i]
        if buf is None or buf.numel() < n_ints:
            buf = torch.empty(max(n_ints, 4096), dtype=torch.int32, pin_memory=True)
            self.host[i] = buf
        return buf, i

    def sent(self, i: int) -> None:
        ev = self.events[i] or torch.cuda.Event()
        ev.record()
        self.events[i] = ev
