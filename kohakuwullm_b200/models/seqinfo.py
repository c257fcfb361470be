"""Sequence layout carried next to the tokens.

Packed layout: ``tokens`` is (T,), ``cu_seqlens`` (N+1,) int32 marks document boundaries,
``position_ids`` (T,) restarts at every document. Padded layout: ``tokens`` is (B,S),
``cu_seqlens`` is ``None`` and ``position_ids`` is (B,S). The backbone is a pure function of
``(tokens, seq_info)``. Reference: src/kohakuwullm/models/components/seqinfo.py:11-85.
"""

from __future__ import annotations

from dataclasses import dataclass, field, replace

import torch


def _version(t: torch.Tensor) -> int | None:
    """Count of the writes into ``t``; None for inference tensors, which have no such count."""
    return None if t.is_inference() else t._version


@dataclass
class SeqInfo:
    cu_seqlens: torch.Tensor | None
    position_ids: torch.Tensor
    max_seqlen: int
    num_seqs: int
    # host copy of the document lengths (kept so FLOP accounting and splitters never sync)
    lengths: tuple[int, ...] | None = None
    # (first position, version of ``position_ids``) when every row is known to count up from one host-known position
    _count: tuple[int, int | None] | None = field(default=None, init=False, repr=False, compare=False)

    def __setattr__(self, name, value):
        if name == "position_ids":
            super().__setattr__("_count", None)
        super().__setattr__(name, value)

    @property
    def start(self) -> int | None:
        """Position of the first column when every row of a padded batch is ``start, start + 1, ...``, known without
        reading the device; None when the positions were given, replaced or written to, or are an inference tensor (whose
        writes torch does not count)."""
        if self._count is None or self._count[1] is None or _version(self.position_ids) != self._count[1]:
            return None
        return self._count[0]

    # a copied or unpickled tensor counts its writes anew, so what is known goes over as the bare position
    def __getstate__(self):
        return {**self.__dict__, "_count": self.start}

    def __setstate__(self, state):
        start = state.get("_count")
        self.__dict__.update(state)
        self._count = None if start is None else (start, _version(self.position_ids))

    @property
    def packed(self) -> bool:
        return self.cu_seqlens is not None

    @property
    def seqlens(self) -> torch.Tensor:
        if self.cu_seqlens is None:
            b, s = self.position_ids.shape
            return torch.full((b,), s, dtype=torch.int32, device=self.position_ids.device)
        return self.cu_seqlens[1:] - self.cu_seqlens[:-1]

    @property
    def total_tokens(self) -> int:
        return int(self.position_ids.numel())

    @classmethod
    def from_lengths(cls, lengths, device=None) -> "SeqInfo":
        lens = [int(x) for x in lengths]
        if any(n <= 0 for n in lens):
            raise ValueError("document lengths must be positive")
        lt = torch.tensor(lens, dtype=torch.int32)
        cu = torch.zeros(len(lens) + 1, dtype=torch.int32)
        cu[1:] = torch.cumsum(lt, 0)
        total = int(cu[-1])
        # position = index - start of its own document
        starts = torch.repeat_interleave(cu[:-1].long(), lt.long())
        pos = torch.arange(total, dtype=torch.long) - starts
        info = cls(cu, pos, max(lens) if lens else 0, len(lens), tuple(lens))
        return info.to(device) if device is not None else info

    @classmethod
    def padded(cls, batch: int, seqlen: int, device=None, offset: int | torch.Tensor = 0) -> "SeqInfo":
        pos = torch.arange(seqlen, dtype=torch.long, device=device).unsqueeze(0).expand(batch, seqlen)
        if isinstance(offset, torch.Tensor):
            pos = pos + offset.to(pos.device).reshape(-1, 1)
        elif offset:
            pos = pos + int(offset)
        info = cls(None, pos, seqlen, batch, None)
        if not isinstance(offset, torch.Tensor):
            info._count = (int(offset), _version(pos))
        return info

    def to(self, device, non_blocking: bool = False) -> "SeqInfo":
        cu = None if self.cu_seqlens is None else self.cu_seqlens.to(device, non_blocking=non_blocking)
        new = replace(self, cu_seqlens=cu, position_ids=self.position_ids.to(device, non_blocking=non_blocking))
        if self.start is not None:
            new._count = (self.start, _version(new.position_ids))
        return new

    def pin_memory(self) -> "SeqInfo":
        cu = None if self.cu_seqlens is None else self.cu_seqlens.pin_memory()
        return replace(self, cu_seqlens=cu, position_ids=self.position_ids.pin_memory())
