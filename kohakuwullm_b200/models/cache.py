"""Key/value cache for incremental decoding (padded layout only).

One (B, max_len, kv_heads, head_dim) K and V buffer per layer, allocated lazily from the first
append. ``static=True`` preallocates ``max_len`` rows and returns the whole buffer with a validity mask
(fixed shapes, CUDA-graph friendly); the dynamic cache returns only the filled prefix. All layers share
one ``length``, advanced by ``advance`` after the last layer of a step. Reference:
src/kohakuwullm/models/cache.py:14-199.
"""

from __future__ import annotations

import torch

from kohakuwullm_b200.models.seqinfo import SeqInfo


class KVCache:
    def __init__(self, num_layers: int, max_len: int, static: bool = True):
        self.num_layers, self.max_len, self.static = num_layers, max_len, static
        self.k: list[torch.Tensor | None] = [None] * num_layers
        self.v: list[torch.Tensor | None] = [None] * num_layers
        self.length = 0
        self._pending = 0
        # while one-token steps are captured: the next position as device integers (int64 for indexing, int32 for the
        # decode kernel), advanced by the step itself
        self.position: tuple[torch.Tensor, torch.Tensor] | None = None

    @classmethod
    def from_config(cls, config, max_len: int, static: bool = True, num_layers: int | None = None):
        return cls(num_layers if num_layers is not None else config.depth, max_len, static)

    def seq_info(self, tokens: torch.Tensor) -> SeqInfo:
        """Layout of the next ``tokens`` (B,S): positions continue after the cached prefix."""
        b, s = tokens.shape
        if self.position is not None:
            return SeqInfo(None, self.position[0].view(1, 1).expand(b, s), s, b, None)
        return SeqInfo.padded(b, s, device=tokens.device, offset=self.length)

    def append(self, layer: int, k: torch.Tensor, v: torch.Tensor, q_pos: torch.Tensor):
        """Store this step's keys/values; returns ``(k_all, v_all, key_positions, key_valid)``."""
        k_all, v_all = self.store(layer, k, v)
        return k_all, v_all, *self.key_positions(k_all, k.shape[1])

    def key_positions(self, k_all: torch.Tensor, new: int):
        """Positions of the keys in ``k_all`` and which of them exist, once ``new`` ones are stored."""
        B, used = k_all.shape[:2]
        pos = torch.arange(used, device=k_all.device)[None, :].expand(B, used)
        return pos, pos < self.length + new

    def store(self, layer: int, k: torch.Tensor, v: torch.Tensor):
        """:meth:`append` for kernels that know which keys exist: returns ``(k_all, v_all)`` alone."""
        B, S = k.shape[:2]
        end = self.length + S
        if end > self.max_len:
            raise RuntimeError(f"KV cache overflow: {end} > max_len {self.max_len}")
        if self.k[layer] is None:
            shape = (B, self.max_len, *k.shape[2:])
            self.k[layer] = torch.zeros(shape, dtype=k.dtype, device=k.device)
            self.v[layer] = torch.zeros(shape, dtype=v.dtype, device=v.device)
        if self.position is not None:
            self.k[layer].index_copy_(1, self.position[0], k)
            self.v[layer].index_copy_(1, self.position[0], v)
            self._pending = S
            return self.k[layer], self.v[layer]
        self.k[layer][:, self.length:end] = k
        self.v[layer][:, self.length:end] = v
        self._pending = S
        used = self.max_len if self.static else end
        return self.k[layer][:, :used], self.v[layer][:, :used]

    def hold_position(self, device) -> None:
        """One-token steps from here on read their position from the device (every buffer exists: a static cache past
        its first step), so that a captured step can be replayed for each next token."""
        self.position = (torch.full((1,), self.length, dtype=torch.int64, device=device),
                         torch.full((1,), self.length, dtype=torch.int32, device=device))

    def advance(self) -> None:
        if self.position is not None:
            for p in self.position:
                p += self._pending
        self.length += self._pending
        self._pending = 0

    def reset(self) -> None:
        self.length = 0
        self._pending = 0
        self.position = None


_APPEND = KVCache.append


def stores_plainly(cache) -> bool:
    """Whether ``cache`` keeps keys and values the way :meth:`KVCache.append` does, so that a kernel may go without the
    positions that it returns. A cache with an ``append`` of its own is asked through it."""
    return getattr(getattr(cache, "append", None), "__func__", None) is _APPEND


def keeps_as_is(buffer: torch.Tensor | None, x: torch.Tensor) -> bool:
    """Whether storing ``x`` (B, S, ...) changes nothing about it: a new buffer, or one of its type and batch size."""
    return buffer is None or (buffer.dtype == x.dtype and buffer.shape[0] == x.shape[0])
