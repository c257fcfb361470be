"""The work whose speed is measured: what users of this framework run, through its public entry points.

Four paths, each over the sizes, data types and options that the shipped configurations use:

``train``     ``TrainEngine.step`` on host-pinned packs: forward, backward, clipping, optimizer, MXFP8 weight refresh
              and router balancing. What a pretraining run repeats for days.
``score``     a packed batch of documents through ``LMBackbone`` and ``LMHead.token_loss`` without gradients:
              validation and per-token log-probabilities.
``prefill``   a batch of long prompts into an empty ``KVCache``: the first step of every decode.
``generate``  ``LocalGenerator.generate`` (cached decode, greedy or sampled), then the new tokens' logits from one packed
              pass over what was written, as a program does that ranks its samples.
"""

from __future__ import annotations

import gc
import math

import torch

from kohakuwullm_b200.data.packing import split_packed
from kohakuwullm_b200.data.synthetic import make_pack, make_packs
from kohakuwullm_b200.generation.engine import LocalGenerator
from kohakuwullm_b200.models import KVCache, LMBackbone, SeqInfo, get_preset
from kohakuwullm_b200.training.engine import TrainEngine
from kohakuwullm_b200.training.optim.lowbit import cast_parameters_

DEVICE = "cuda"

# learning rates of the shipped recipes; Muon's own rate is configs/lm/tipo/tipo_500m.py's
LR, MUON_LR = 3e-4, 0.02


def listed() -> list[dict]:
    return [
        # the debug recipe (configs/lm/smoke/debug.py): tiny kernels, so launches and host work are what counts
        {"name": "train_smoke", "path": "train", "preset": "B200-smoke", "mxfp8": False, "optimizer": "fused_adamw",
         "micro": 2, "tokens": 1024, "split": False, "doc_min": 16, "doc_max": 512, "log_docs": False},
        # the headline benchmark: dense 546M in MXFP8, 4 packs of 4096 tokens a step
        {"name": "train_dense_546m", "path": "train", "preset": "B200-dense-546M", "mxfp8": True, "optimizer": "fused_adamw",
         "micro": 4, "tokens": 4096, "split": False, "doc_min": 64, "doc_max": 4096, "log_docs": False},
        # 64 experts, top-6, MXFP8 expert products, 4 packs of 8192 tokens (configs/lm/moe_991m_ddp.py)
        {"name": "train_moe_991m", "path": "train", "preset": "B200-moe-991M", "mxfp8": True, "optimizer": "fused_adamw",
         "micro": 4, "tokens": 8192, "split": False, "doc_min": 64, "doc_max": 4096, "log_docs": False},
        # 1.1B in bf16 with sliding windows, four sinks a head and YaRN, one long pack (configs/lm/sliding_1b.py)
        {"name": "train_sliding_1b", "path": "train", "preset": "B200-sliding-1B", "mxfp8": False, "optimizer": "fused_adamw",
         "micro": 1, "tokens": 16384, "split": False, "doc_min": 128, "doc_max": 16384, "log_docs": True},
        # short captions, Muon, a batch split at document boundaries into two uneven micro-batches (configs/lm/tipo/tipo_500m.py)
        {"name": "train_500m_muon_ragged", "path": "train", "preset": "Kohaku-500M", "mxfp8": True, "optimizer": "muon",
         "micro": 2, "tokens": 5003, "split": True, "doc_min": 50, "doc_max": 600, "log_docs": False},
        # top-8 routing in plain bf16, uneven micro-batches: the presets' own default precision
        {"name": "train_moe_1b_bf16", "path": "train", "preset": "Kohaku-MoE-1B", "mxfp8": False, "optimizer": "fused_adamw",
         "micro": 2, "tokens": 3001, "split": True, "doc_min": 32, "doc_max": 1024, "log_docs": True},
        # validation on one odd-sized pack
        {"name": "score_500m", "path": "score", "preset": "Kohaku-500M", "mxfp8": False, "tokens": 8190, "doc_min": 32,
         "doc_max": 2048, "log_docs": True},
        # the same on a routed model, a small pack
        {"name": "score_moe_1b", "path": "score", "preset": "Kohaku-MoE-1B", "mxfp8": False, "tokens": 1500, "doc_min": 32,
         "doc_max": 1024, "log_docs": True},
        # two long prompts
        {"name": "prefill_546m", "path": "prefill", "preset": "B200-dense-546M", "mxfp8": False, "rows": 2, "prompt": 3001},
        # one short prompt, greedy: the interactive case (the smallest decode there is)
        {"name": "generate_200m_greedy", "path": "generate", "preset": "Kohaku-200M", "mxfp8": False, "rows": 1, "prompt": 23,
         "new": 48, "temperature": 0.0, "top_p": 1.0},
        # cli/sample.py's defaults with several samples of a prompt
        {"name": "generate_500m_sampled", "path": "generate", "preset": "Kohaku-500M", "mxfp8": False, "rows": 8, "prompt": 200,
         "new": 32, "temperature": 0.8, "top_p": 0.95},
        # in-training preview of the routed recipe (configs/lm/general/general_1b.py samples at temperature 1)
        {"name": "generate_moe_1b", "path": "generate", "preset": "Kohaku-MoE-1B", "mxfp8": False, "rows": 2, "prompt": 64,
         "new": 24, "temperature": 1.0, "top_p": 1.0},
    ]


# ------------------------------------------------------------------------------------ drawn cases
def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    path = rng.choice(["train", "train", "train", "score", "prefill", "generate", "generate"])
    if path == "train":
        preset, mxfp8 = rng.choice([("B200-smoke", False), ("Kohaku-200M", False), ("Kohaku-200M", True), ("Kohaku-500M", False),
                                    ("Kohaku-500M", True), ("B200-dense-546M", True), ("B200-moe-991M", True),
                                    ("Kohaku-MoE-1B", False), ("Kohaku-MoE-1B", True), ("B200-sliding-1B", False)])
        split = rng.random() < 0.5
        tokens = _log_int(rng, 512, 4096 if split else 8192)     # a split batch captures a graph for each size that it makes
        muon = preset != "B200-smoke" and rng.random() < 0.25
        case = {"path": path, "preset": preset, "mxfp8": mxfp8, "optimizer": "muon" if muon else "fused_adamw",
                "micro": rng.randint(1, 4), "tokens": tokens, "split": split, "doc_min": rng.randint(16, 64),
                "doc_max": _log_int(rng, 128, tokens), "log_docs": rng.random() < 0.5}
        while case["micro"] > 1 and work(case)["flops"] > 9e13:  # train_sliding_1b's, the largest listed
            case["micro"] -= 1
        return case
    preset = rng.choice(["Kohaku-200M", "Kohaku-500M", "B200-dense-546M", "Kohaku-MoE-1B", "B200-sliding-1B"])
    if path == "score":
        tokens = _log_int(rng, 100, 16384)
        return {"path": path, "preset": preset, "mxfp8": False, "tokens": tokens, "doc_min": 16, "doc_max": _log_int(rng, 64, 4096),
                "log_docs": rng.random() < 0.5}
    if path == "prefill":
        prompt = _log_int(rng, 64, 3500)
        return {"path": path, "preset": preset, "mxfp8": False, "rows": rng.randint(1, 4 if prompt < 2000 else 2), "prompt": prompt}
    temperature, top_p = rng.choice([(0.0, 1.0), (0.8, 0.95), (1.0, 1.0)])
    return {"path": path, "preset": preset, "mxfp8": False, "rows": _log_int(rng, 1, 16), "prompt": _log_int(rng, 8, 512),
            "new": rng.randint(8, 48), "temperature": temperature, "top_p": top_p}


# ------------------------------------------------------------------------------------ inputs
def _model(case: dict, seed: int) -> LMBackbone:
    torch.manual_seed(seed)
    with torch.device(DEVICE):
        return LMBackbone(get_preset(case["preset"], mxfp8=case["mxfp8"]))


@torch.no_grad()
def _decided(model: LMBackbone) -> None:
    """Weights of a trained model's kind. Fresh random weights leave the next token a near tie between 65536 ids, and
    rounding would pick it; a trained model is sure of most tokens. Here the residual stream keeps a clear trace of the
    token and the head reads its successor from it, so one id stands clear of the rest while every block still
    contributes to the hidden state and the logits."""
    table = model.embed.weight
    table.normal_(0.0, 0.25)
    model.head.weight.copy_(table.roll(1, 0) * (6.0 / math.sqrt(table.shape[1])))


def prepare(case: dict, seed: int) -> dict:
    gc.collect()        # an engine of an earlier call and its CUDA graphs hold each other
    model = _model(case, seed)
    cfg = model.config
    gen = torch.Generator().manual_seed(seed)
    if case["path"] == "train":
        kw = {"optimizer_kwargs": {"muon_lr": MUON_LR}} if case["optimizer"] == "muon" else {}
        engine = TrainEngine(model, lr=LR, param_dtype=torch.bfloat16, optimizer=case["optimizer"], **kw)
        docs = (case["doc_min"], case["doc_max"], cfg.vocab_size, seed, case["log_docs"])
        if case["split"]:
            packs = split_packed(make_pack(case["micro"] * case["tokens"], *docs), case["micro"])
        else:
            packs = make_packs(case["micro"], case["tokens"], *docs)
        return {"case": case, "engine": engine, "packs": [p.pin_memory() for p in packs]}
    _decided(model)
    cast_parameters_(model, torch.bfloat16)
    model.eval()
    if case["path"] == "score":
        pack = make_pack(case["tokens"], case["doc_min"], case["doc_max"], cfg.vocab_size, seed, case["log_docs"])
        return {"case": case, "model": model, "pack": pack.to(DEVICE)}
    # ids below 60000: a greedy walk of 48 successors does not run into the end of the vocabulary (and EOS, id 0)
    prompt = torch.randint(1, 60000, (case["rows"], case["prompt"]), generator=gen).to(DEVICE)
    if case["path"] == "prefill":
        return {"case": case, "model": model, "prompt": prompt}
    return {"case": case, "model": model, "prompt": prompt, "generator": LocalGenerator(model, eos_id=0)}


# ------------------------------------------------------------------------------------ one pass
def run(state: dict):
    case = state["case"]
    if case["path"] == "train":
        engine = state["engine"]
        out = engine.step(state["packs"])
        # weights and not gradients: a router's near ties and e4m3 rounding make single gradient values a matter of
        # the last bit in any implementation, while the step that the weights take is well defined
        return {"loss": out["loss"], "ce": out["ce"], "grad_norm": out["grad_norm"],
                "weights": {key: group.data for key, group in engine.flat.groups.items()}}
    model = state["model"]
    with torch.no_grad():
        if case["path"] == "score":
            pack = state["pack"]
            hidden = model(pack.tokens, pack.seq_info)
            ce, lse = model.head.token_loss(hidden, pack.labels)
            return {"hidden": hidden, "ce": ce, "lse": lse}
        prompt = state["prompt"]
        rows, length = prompt.shape
        if case["path"] == "prefill":
            cache = KVCache.from_config(model.config, length + 64)
            hidden = model(prompt, cache.seq_info(prompt), cache=cache)
            logits = model.head.logits(hidden[:, -1])
            return {"hidden": hidden, "logits": logits, "k": [k[:, :length] for k in cache.k],
                    "v": [v[:, :length] for v in cache.v]}
        tokens = state["generator"].generate(prompt, case["new"], temperature=case["temperature"], top_p=case["top_p"])
        total = tokens.shape[1]
        hidden = model(tokens.reshape(-1), SeqInfo.from_lengths([total] * rows, device=tokens.device))
        return {"tokens": tokens, "logits": model.head.logits(hidden.view(rows, total, -1)[:, length - 1:-1])}


# ------------------------------------------------------------------------------------ what a pass cannot do without
def _sizes(cfg):
    """(parameters, parameters of the matrix products that one token goes through) without the embedding's lookup."""
    attn = cfg.dim * (cfg.heads + 2 * cfg.kv_heads) * cfg.head_dim + cfg.heads * cfg.head_dim * cfg.dim
    dense = 3 * cfg.dim * (cfg.mlp_hidden or 0)
    total = active = cfg.dim * cfg.vocab_size                # the head
    for routed in cfg.moe_layers:
        total, active = total + attn, active + attn
        if routed:
            expert = 3 * cfg.dim * cfg.moe_hidden
            total += expert * (cfg.moe_num_experts + cfg.moe_num_shared) + cfg.dim * cfg.moe_num_experts
            active += expert * (cfg.moe_top_k + cfg.moe_num_shared) + cfg.dim * cfg.moe_num_experts
        else:
            total, active = total + dense, active + dense
    return total + cfg.dim * cfg.vocab_size, active


def _attention_flops(cfg, length: float) -> float:
    """Forward attention products per token of a document of ``length``: two products over the causal half or window."""
    pairs = sum(min(w or length, length) if w else length / 2 for w in cfg.windows)
    return 4.0 * pairs * cfg.heads * cfg.head_dim


def work(case: dict) -> dict:
    cfg = get_preset(case["preset"], mxfp8=case["mxfp8"])
    total, active = _sizes(cfg)
    if case["path"] == "train":
        tokens = case["micro"] * case["tokens"]
        length = min((case["doc_min"] + case["doc_max"]) / 2, case["tokens"])
        # weights, fp32 masters and both moments in and out (Muon: 16-bit weights and momentum); gradients stay in the step
        state = 28 if case["optimizer"] == "fused_adamw" else 8
        return {"bytes": total * state + tokens * 24, "flops": tokens * (6.0 * active + 3.5 * _attention_flops(cfg, length))}
    if case["path"] == "score":
        n = case["tokens"]
        length = min((case["doc_min"] + case["doc_max"]) / 2, n)
        return {"bytes": 2 * total + n * (2 * cfg.dim + 32), "flops": n * (2.0 * active + _attention_flops(cfg, length))}
    rows, prompt = case["rows"], case["prompt"]
    kv = 4 * cfg.depth * cfg.kv_heads * cfg.head_dim            # bytes of keys and values of one position
    body = active - cfg.dim * cfg.vocab_size
    if case["path"] == "prefill":
        n = rows * prompt
        return {"bytes": 2 * total + n * (kv + 2 * cfg.dim + 8) + 4 * rows * cfg.vocab_size,
                "flops": n * (2.0 * body + _attention_flops(cfg, prompt)) + 2.0 * rows * cfg.dim * cfg.vocab_size}
    new = case["new"]
    # every new token reads the weights its rows go through and their cached keys and values; then one pass over all
    step = 2 * min(total, body * rows if any(cfg.moe_layers) else body) + 2 * cfg.dim * cfg.vocab_size
    reads = rows * kv * (prompt + new / 2)
    n = rows * (prompt + new)
    return {"bytes": new * (step + reads) + 2 * total + 4 * rows * new * cfg.vocab_size,
            "flops": 2.0 * n * (2.0 * body) + 4.0 * rows * new * cfg.dim * cfg.vocab_size}


def tolerance(case: dict) -> dict:
    """Measured by running each path with its attention replaced by the fp32 explicit-mask form (same bf16 storage, other
    sums and roundings) and, for ``prefill``, by running the prompt as packed documents: the second step's weights differ by
    0.007 to 0.014 (e4m3 rounding, routing ties and Adam's division by the gradient's own size amplify the last bit), hidden
    states and logits by 0.009 to 0.015 after 16 to 24 layers. The tokens are the same."""
    return {"rel": 0.03}
