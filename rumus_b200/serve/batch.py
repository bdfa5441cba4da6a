"""What one engine step computes: some tokens of some sequences, as one ragged batch."""
from __future__ import annotations

from dataclasses import dataclass, replace
from typing import List, Optional

import torch


@dataclass
class Portion:
    """The next tokens of one sequence: ``tokens`` stand at positions ``start ...``; ``want``: the places
    among them whose logits are asked for."""
    rid: int
    start: int
    tokens: List[int]
    want: List[int]


@dataclass
class Segment:
    """A prompt portion inside the batch: rows ``row0 .. row0 + n`` are tokens ``start .. start + n``."""
    start: int
    n: int
    row0: int


@dataclass
class StepBatch:
    """Rows ``0 .. n_rows`` are single tokens that attend through their own block table and context length
    (decoded tokens, and the tokens of portions too short for a tile of queries); the ``segments`` follow.
    Nothing a model reads on the host depends on the first kind beyond ``n_rows`` and ``max_ctx``, so a step
    without segments can be captured as a CUDA graph."""
    tokens: torch.Tensor                 # int64 [T]
    positions: torch.Tensor              # int64 [T]
    slots: torch.Tensor                  # int64 [T] cache slot of every token, -1 = keep nothing
    n_rows: int
    tables: Optional[torch.Tensor]       # int32 [n_rows, max_blocks]
    ctx: Optional[torch.Tensor]          # int32 [n_rows] keys the row sees, its own included
    max_ctx: int                         # no entry of ctx is larger
    segments: List[Segment]
    seg_tables: Optional[torch.Tensor]   # int32 [len(segments), max_blocks]
    # The portions themselves, for models with state per sequence: (first row, tokens, place of the sequence, position
    # of the first token).  The first ``n_short`` stand in the single rows, the segments follow; no tokens: padding.
    seqs: Optional[torch.Tensor] = None      # int32 [n_short + len(segments), 4]
    n_short: int = 0
    wanted: Optional[torch.Tensor] = None    # int64: rows whose logits are asked for, in the caller's order

    def to(self, device) -> "StepBatch":
        """The same batch with its tensors on ``device``: one copy of them all, which waits for nothing on a GPU."""
        names = [n for n in ("tokens", "positions", "slots", "wanted", "tables", "ctx", "seg_tables", "seqs") if getattr(self, n) is not None]
        parts = [getattr(self, n) for n in names]
        sizes = [t.numel() * t.element_size() // 4 for t in parts]        # in int32
        room = [-(-k // 64) * 64 for k in sizes]                           # every tensor starts on a 256-byte boundary

        def views(flat):
            return [piece[:k].view(t.dtype).view(t.shape) for piece, k, t in zip(flat.split(room), sizes, parts)]

        host = torch.empty(sum(room), dtype=torch.int32, pin_memory=torch.device(device).type == "cuda")
        for view, t in zip(views(host), parts):
            view.copy_(t)
        return replace(self, **dict(zip(names, views(host.to(device, non_blocking=True)))))


def to_device(numbers, device, dtype=torch.int32) -> torch.Tensor:
    """A list of numbers on ``device``, without waiting for what runs there (a copy from pageable memory would)."""
    return torch.tensor(numbers, dtype=dtype, pin_memory=torch.device(device).type == "cuda").to(device, non_blocking=True)
