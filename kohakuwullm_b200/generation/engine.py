"""Text generation: sampling filters, single-process and pipelined generators.

Sampling is done in fp32 with the filters applied in the order top-k -> top-p -> min-p, greedy when
``temperature <= 0``; the generator owns a private per-device RNG (``SAMPLE_SEED``) so sampling never
perturbs the training RNG stream. Rows that have emitted a stop id keep emitting EOS.
``LocalGenerator`` decodes with a static KV cache (``use_cache=False`` recomputes the whole prefix each
step: the reference path used by the equivalence tests). ``PipelineGenerator`` decodes through the stages
of a pipeline: rank 0 embeds and runs its blocks, every rank forwards the ``(rows, S, dim)`` hidden state
to the next with NCCL send/recv, the last rank samples and broadcasts the next token. With
``microbatches=m`` the rows are cut into m chunks, each with a KV cache of its own on every stage, and one
decode step runs the chunks through the stages as a forward-only GPipe wave (sends are asynchronous, so stage
s works on chunk c + 1 while stage s + 1 works on chunk c); the last stage samples all rows at once, so the
tokens do not depend on m. ``max_new_tokens=None`` decodes until every row has stopped or the context is full.
Reference: src/kohakuwullm/generation/engine.py:19-385.
"""

from __future__ import annotations

import ctypes
import warnings
from typing import Sequence

import torch
import torch.distributed as dist

from kohakuwullm_b200.models.cache import KVCache
from kohakuwullm_b200.models.seqinfo import SeqInfo
from kohakuwullm_b200.ops import native
from kohakuwullm_b200.ops.mxfp8 import clear_prequantized

SAMPLE_SEED = 20090220


def filter_top_k(logits: torch.Tensor, k: int) -> torch.Tensor:
    if k <= 0 or k >= logits.shape[-1]:
        return logits
    kth = logits.topk(k, dim=-1).values[..., -1:]
    return logits.masked_fill(logits < kth, float("-inf"))


def filter_top_p(logits: torch.Tensor, p: float) -> torch.Tensor:
    if p >= 1.0:
        return logits
    sorted_logits, order = logits.sort(dim=-1, descending=True)
    probs = sorted_logits.softmax(-1)
    cum = probs.cumsum(-1)
    drop = (cum - probs) >= p           # keep the token that crosses the threshold
    sorted_logits = sorted_logits.masked_fill(drop, float("-inf"))
    return torch.full_like(logits, float("-inf")).scatter(-1, order, sorted_logits)


def filter_min_p(logits: torch.Tensor, min_p: float) -> torch.Tensor:
    if min_p <= 0.0:
        return logits
    probs = logits.softmax(-1)
    floor = probs.max(-1, keepdim=True).values * min_p
    return logits.masked_fill(probs < floor, float("-inf"))


def sample(logits: torch.Tensor, temperature: float = 1.0, top_k: int = 0, top_p: float = 1.0,
           min_p: float = 0.0, generator: torch.Generator | None = None) -> torch.Tensor:
    """logits (rows, vocab) -> next ids (rows,)."""
    logits = logits.float()
    if not torch.isfinite(logits).any(-1).all():
        raise FloatingPointError("non-finite logits reached the sampler")
    if temperature <= 0:
        return logits.argmax(-1)
    logits = logits / temperature
    logits = filter_min_p(filter_top_p(filter_top_k(logits, top_k), top_p), min_p)
    return torch.multinomial(logits.softmax(-1), 1, generator=generator).squeeze(-1)


def token_budget(max_new_tokens: int | None, prompt_len: int, max_position: int) -> int:
    """New tokens to decode: the request, cut to what the model's context still holds (None: all of it)."""
    room = max(int(max_position) - int(prompt_len), 0)
    if max_new_tokens is None:
        return room
    # an explicit request is honoured up to the context; a prompt that already fills the context keeps the request
    # (rotary positions extrapolate; the caller asked for it)
    return min(int(max_new_tokens), room) if room else int(max_new_tokens)


def advance(tokens: torch.Tensor, nxt: torch.Tensor, finished: torch.Tensor, stop_ids: Sequence[int], eos: int):
    """Append ``nxt``; rows that already finished are held at EOS. Returns (tokens, finished)."""
    nxt = torch.where(finished, torch.full_like(nxt, eos), nxt)
    hit = torch.zeros_like(finished)
    for s in stop_ids:
        hit |= nxt == s
    return torch.cat([tokens, nxt[:, None]], dim=1), finished | hit


class CapturePool:
    """Memory and stream of captured steps, one capture at a time: the next one takes over what the last one has left."""

    def __init__(self, device):
        self.lib, handle = native.require(), ctypes.c_void_p()
        with torch.cuda.device(device):
            self.memory = torch.cuda.MemPool()
            native.check(self.lib.kwu_stream_create(ctypes.byref(handle)), "stream of decode captures")
        # blocks of the memory belong to the stream that they were made on
        self.stream = torch.cuda.ExternalStream(handle.value, device=device)

    def __del__(self):
        if getattr(self, "stream", None) is not None:
            self.lib.kwu_stream_destroy(ctypes.c_void_p(self.stream.cuda_stream))


class StepGraph:
    """One cached decode step (embedding to logits of one new token a row) captured as a CUDA graph.

    A step is 15 to 20 short kernels a layer; issued from Python they leave the GPU idle for most of the step, replayed
    they follow each other. The position lives on the device (``KVCache.hold_position``), so one capture serves every
    remaining token of the call. The capture is the library's own and not torch's, whose captures make every other thread's
    draw from the device's default generator fail for as long as they last."""

    MIN_STEPS = 3     # a capture costs about a step issued from Python, so it pays from the third on

    def __init__(self, backbone, cache, token: torch.Tensor, pool: CapturePool):
        self.lib, self.exec = native.require(), ctypes.c_void_p()
        self.token = token.clone()
        length = cache.length
        cache.hold_position(token.device)
        handle = ctypes.c_void_p(pool.stream.cuda_stream)
        pool.stream.wait_stream(torch.cuda.current_stream(token.device))
        try:
            with torch.cuda.stream(pool.stream), torch.cuda.use_mem_pool(pool.memory, token.device):
                native.check(self.lib.kwu_capture_begin(handle), "capture of a decode step")
                exec_at = None
                try:
                    hidden = backbone(self.token, cache.seq_info(self.token), cache=cache)
                    self.logits = backbone.head.logits(hidden[:, -1])
                    exec_at = ctypes.byref(self.exec)
                finally:
                    rc = self.lib.kwu_capture_end(handle, exec_at)     # also ends a capture that failed on the way
                native.check(rc, "capture of a decode step")
        except BaseException:
            cache.position = None
            raise
        finally:
            cache.length, cache._pending = length, 0      # nothing has run yet
            if backbone.config.mxfp8:
                clear_prequantized()                       # copies that the capture has made and nothing took

    def __call__(self, cache, token: torch.Tensor) -> torch.Tensor:
        if cache.length + 1 > cache.max_len:
            raise RuntimeError(f"KV cache overflow: {cache.length + 1} > max_len {cache.max_len}")
        self.token.copy_(token)
        native.check(self.lib.kwu_graph_launch(self.exec, native.stream_ptr()), "decode step")
        cache.length += 1
        return self.logits

    def __del__(self):
        if getattr(self, "exec", None):
            self.lib.kwu_graph_destroy(self.exec)


def capturable(backbone, tokens: torch.Tensor) -> bool:
    """Whether a cached one-token step of this model is a fixed sequence of kernels: every module is one whose decode path
    reads nothing back to the host, runs on the native kernels, and carries no hooks, modes or replaced methods that a
    replay would skip."""
    from torch.nn.modules import module as hooks

    from kohakuwullm_b200.models.backbone import LMBackbone
    from kohakuwullm_b200.models.block import DecoderBlock
    from kohakuwullm_b200.models.components import attention, mlp, moe, norm, posenc
    from kohakuwullm_b200.models.head import LMHead

    plain = (LMBackbone, DecoderBlock, LMHead, mlp.Linear, mlp.GLUMLP, mlp.GeGLUMLP, mlp.GELUMLP, norm.RMSNorm,
             norm.GemmaRMSNorm, norm.LayerNorm, norm.DyT, posenc.RoPE, posenc.NoPE, torch.nn.Embedding, torch.nn.ModuleList,
             torch.nn.Identity)
    if type(backbone) is not LMBackbone or not tokens.is_cuda or not native.available() \
            or torch.cuda.is_current_stream_capturing() or hooks._global_forward_hooks or hooks._global_forward_pre_hooks:
        return False
    # dispatch and function modes (operation counters, loggers) see every operator of a step issued directly
    if torch._C._len_torch_dispatch_stack() or torch._C._len_torch_function_stack():
        return False
    if backbone.embed.weight.dtype != torch.bfloat16 or backbone.config.head_dim != 64:
        return False
    if any(t.device != tokens.device for group in (backbone.parameters(), backbone.buffers()) for t in group):
        return False
    for m in backbone.modules():
        if m._forward_hooks or m._forward_pre_hooks or any(callable(v) for v in vars(m).values()):
            return False
        if type(m) is attention.Attention:
            if m.heads % m.kv_heads or m.heads // m.kv_heads > 8 or \
                    not (m.qk_norm or type(backbone.pos_enc) is posenc.RoPE):     # q would be a view of the projection
                return False
        elif type(m) is moe.MoEMLP:
            w = m.router.weight
            if m.ep_world > 1 or m.expert_path not in (None, "grouped") or type(m.router) is not moe.TopKRouter \
                    or m.router.num_groups > 1 or w.shape[0] > 128 or w.shape[0] % 8 or w.dtype != torch.float32 \
                    or m.w_in.dtype != torch.bfloat16 or m.dim % 64 or m.w_in.shape[1] % 128:
                return False
        elif type(m) is not moe.TopKRouter and type(m) not in plain:
            return False
    return True


class LocalGenerator:
    def __init__(self, backbone, eos_id: int = 0, stop_ids: Sequence[int] = (), use_cache: bool = True,
                 static_cache: bool = True):
        self.backbone, self.eos = backbone, eos_id
        self.stop_ids = tuple(stop_ids) or (eos_id,)
        self.use_cache, self.static_cache = use_cache, static_cache
        self._rng: dict[str, torch.Generator] = {}
        self._pools: dict[str, CapturePool] = {}      # what the last finished call on a device captured into

    def rng(self, device) -> torch.Generator:
        key = str(device)
        if key not in self._rng:
            self._rng[key] = torch.Generator(device=device).manual_seed(SAMPLE_SEED)
        return self._rng[key]

    @torch.no_grad()
    def generate(self, prompt: torch.Tensor, max_new_tokens: int | None = 128, **sampling) -> torch.Tensor:
        """prompt (rows, S) of equal-length rows -> (rows, S + new). ``max_new_tokens=None``: until every row has
        stopped or the context is full."""
        bb = self.backbone
        max_new_tokens = token_budget(max_new_tokens, prompt.shape[1], getattr(bb.config, "max_position", 1 << 30))
        was_training = bb.training
        bb.eval()
        tokens = prompt
        rows, S = prompt.shape
        finished = torch.zeros(rows, dtype=torch.bool, device=prompt.device)
        gen = self.rng(prompt.device)
        cache = KVCache.from_config(bb.config, S + max_new_tokens, static=self.static_cache) if self.use_cache else None
        step_in = prompt
        graph, pool, graphs = None, None, cache is not None and self.static_cache and capturable(bb, prompt)
        for i in range(max_new_tokens):
            # the first one-token step is issued directly: it loads kernels and builds what later ones find
            if graphs and graph is None and i >= 2 and max_new_tokens - i >= StepGraph.MIN_STEPS:
                try:
                    # taken out for the call: calls from several threads have a pool each
                    pool = self._pools.pop(str(prompt.device), None) or CapturePool(prompt.device)
                    graph = StepGraph(bb, cache, step_in, pool)
                except RuntimeError as err:    # what cannot be captured is issued directly, and raises there if it is wrong
                    warnings.warn(f"decode steps are issued one by one, their capture failed: {err}")
                    graphs = False
            if graph is not None:
                logits = graph(cache, step_in)
            else:
                if cache is not None:
                    hidden = bb(step_in, cache.seq_info(step_in), cache=cache)
                else:
                    hidden = bb(tokens, SeqInfo.padded(rows, tokens.shape[1], device=tokens.device))
                logits = bb.head.logits(hidden[:, -1])
            nxt = sample(logits, generator=gen, **sampling)
            tokens, finished = advance(tokens, nxt, finished, self.stop_ids, self.eos)
            step_in = tokens[:, -1:]
            if bool(finished.all()):
                break
        if graph is not None:
            self._pools[str(prompt.device)] = pool
        bb.train(was_training)
        return tokens


class PipelineGenerator:
    """Forward-only pipelined decode over ``LMStage`` slices: one KV cache per stage and micro-batch."""

    def __init__(self, stage, rank: int, world: int, eos_id: int = 0, stop_ids: Sequence[int] = (), group=None,
                 microbatches: int | None = None):
        self.stage, self.rank, self.world, self.group = stage, rank, world, group
        self.eos = eos_id
        self.stop_ids = tuple(stop_ids) or (eos_id,)
        self.microbatches = microbatches
        self._gen: torch.Generator | None = None

    def _forward(self, step_in, cache, rows, S, device, dtype, pending):
        """One chunk through this rank's blocks. Returns the last stage's logits of the final position."""
        stage = self.stage
        info = cache.seq_info(torch.empty(rows, S, device=device))
        if stage.is_first:
            x = stage.embed(step_in)
            if stage.embed_scale != 1.0:
                x = x * stage.embed_scale
        else:
            x = torch.empty(rows, S, stage.config.dim, device=device, dtype=dtype)
            dist.recv(x, src=self.rank - 1, group=self.group)
        rope = stage.pos_enc.prepare(info.position_ids)
        for i, blk in enumerate(stage.blocks):
            x = blk(x, info, rope, cache=cache, layer=i)
        cache.advance()
        if stage.is_last:
            return stage.head.logits(stage.final_norm(x)[:, -1])
        x = x.contiguous()
        # asynchronous: this rank goes on with its next chunk while the next stage takes this one
        pending.append((dist.isend(x, dst=self.rank + 1, group=self.group), x))
        return None

    @torch.no_grad()
    def generate(self, prompt: torch.Tensor, max_new_tokens: int | None = 128, **sampling) -> torch.Tensor:
        stage = self.stage
        stage.eval()
        device = prompt.device
        dtype = next(p for p in stage.parameters() if p.dim() >= 2).dtype
        rows, S = prompt.shape
        chunks = self.microbatches or 1
        if rows % chunks:
            raise ValueError(f"{rows} rows do not split into {chunks} micro-batches")
        per = rows // chunks
        budget = token_budget(max_new_tokens, S, getattr(stage.config, "max_position", S + (max_new_tokens or 0)))
        caches = [KVCache(len(stage.blocks), S + budget, static=True) for _ in range(chunks)]
        if self._gen is None:
            self._gen = torch.Generator(device=device).manual_seed(SAMPLE_SEED)
        tokens = prompt
        finished = torch.zeros(rows, dtype=torch.bool, device=device)
        step_in = prompt
        last = self.world - 1
        for _ in range(budget):
            pending: list = []
            logits = [self._forward(step_in[c * per:(c + 1) * per], caches[c], per, step_in.shape[1], device, dtype,
                                    pending) for c in range(chunks)]
            for work, _buf in pending:
                work.wait()
            # all rows are sampled in one call: the random stream is consumed as without micro-batches
            nxt = sample(torch.cat(logits), generator=self._gen, **sampling) if self.rank == last else \
                torch.empty(rows, dtype=torch.long, device=device)
            if self.world > 1:
                dist.broadcast(nxt, src=last, group=self.group)
            tokens, finished = advance(tokens, nxt, finished, self.stop_ids, self.eos)
            step_in = tokens[:, -1:]
            if bool(finished.all()):
                break
        return tokens


def build_generator(model, **kw):
    """``LMBackbone`` -> ``LocalGenerator``; an ``LMStage`` needs ``rank`` and ``world`` -> ``PipelineGenerator``."""
    if hasattr(model, "plan"):
        return PipelineGenerator(model, **kw)
    return LocalGenerator(model, **kw)
