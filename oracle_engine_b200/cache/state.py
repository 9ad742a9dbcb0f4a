"""Per-sequence state of fixed size, beside the cache: one row per slot.

Parts that keep state which does not grow with the sequence (a recurrent or
convolutional mixer's state, for instance) declare it with `state_need()`; the sampler
keeps its random-number counter and its window of recent tokens here too.  Each declared
tensor is stored as [slots, *shape] on the device and its row is zeroed when a slot is
handed to a new sequence.  The Llama decoder's own mixers declare none.

In the reference this is loop state of `Engine::generate` and members of `Sampler`
(core/engine.cpp:118-138, core/sampler.hpp:41-43).
"""
from __future__ import annotations

import torch

from ..csrc import ops


class StateStore:
    def __init__(self, n_slots: int, device):
        self.n_slots = n_slots
        self.device = device
        self._tensors: dict[tuple, torch.Tensor] = {}
        self._rows = None            # (addresses and row sizes of the tensors on the device, the largest row's bytes)

    def add(self, owner, name: str, need) -> torch.Tensor:
        key = (owner, name)
        if key in self._tensors:
            raise ValueError(f"state {key} is declared twice")
        t = torch.zeros((self.n_slots, *need.shape), dtype=need.dtype, device=self.device)
        self._tensors[key] = t
        self._rows = None
        return t

    def views(self, owner) -> dict[str, torch.Tensor]:
        return {name: t for (o, name), t in self._tensors.items() if o == owner}

    def get(self, owner, name: str) -> torch.Tensor:
        return self._tensors[(owner, name)]

    def reset(self, slot: int) -> None:
        """Zeroes the slot's row of every tensor; on the device in one launch (a fill per tensor cost a request of a
        decoder with recurrent layers 0.1 ms of host time, ten times what the memory needs; for the sampler's four tensors
        alone it makes no difference, a 41-token request of the 3B shape 35.58 ms with fills and 35.56 with the launch)."""
        if not 0 <= slot < self.n_slots:
            raise IndexError(f"slot {slot} of {self.n_slots}")
        if self._rows is not None:
            ops.zero_rows(*self._rows, slot)
            return
        tensors = list(self._tensors.values())
        if not tensors:
            return
        if not tensors[0].is_cuda or any(t[0].numel() * t.element_size() % 4 for t in tensors):
            for t in tensors:
                t[slot].zero_()
            return
        self._rows = ops.row_table(tensors)
        ops.zero_rows(*self._rows, slot)

    def total_bytes(self) -> int:
        return sum(t.numel() * t.element_size() for t in self._tensors.values())
