"""``MuonW``: Muon (momentum + Newton-Schulz orthogonalisation) for hidden matrices, 16-bit-state AdamW for
everything else.

Orthogonalisation. For a matrix ``X`` (n, m), n <= m (taller matrices are handled through their transpose),
scaled into the iteration's convergence radius, two iterations are offered:

* ``quintic``  ``X <- a X + (b G + c G G) X`` with ``G = X X^T`` and the fixed coefficients
  (3.4445, -4.7750, 2.0315): three products per step.
* ``cubic5``   five steps ``X <- (a_k I + b_k G) X`` with a per-step schedule: two products per step. Steps can
  be chained in GRAM SPACE: with ``S = a I + b G`` the next Gram matrix is ``S G S`` (n x n products only), so a
  phase of L steps needs one Gram product, 2 (L - 1) small products and ONE n x m product. Shapes whose aspect
  ratio m / n is at least ``gram_aspect`` use the phases (2, 3); squarer ones run the five steps directly.

Batching. All matrices of one shape (the q/k/v/o, MLP and stacked expert weights of every layer) are stacked
and orthogonalised as ONE batch per product, up to ``ns_batch_elems`` elements at a time. On a B200 a product of the
whole batch is one launch of the tcgen05 GEMM over equal matrices (``kwu_gemm_bf16_batched``), without transposes:
``X X^T`` and ``G G`` take both operands K-major, ``P X`` takes X MN-major, and the product that makes a phase's last
``G`` writes ``a I + b G`` in its place. Elsewhere ``torch.bmm``.

Write-back: ``p <- p (1 - lr wd) - lr scale U`` with ``scale`` = ``sqrt(max(1, rows / cols))`` (``spectral``) or
``rms_target sqrt(max(rows, cols))`` (``rms``); ``rounding="stochastic"`` rounds the bf16 result stochastically
(Philox stream, offset advancing by each parameter's element count so the stream does not depend on batching).
Reference: src/kohakuwullm/training/optim/muon.py:20-107 (iterations), :178-442 (optimizer).
"""

from __future__ import annotations

import ctypes
import math

import torch

from kohakuwullm_b200.ops import native
from kohakuwullm_b200.ops.optim import adamw16_step_, sr_update_

ci, cf = ctypes.c_int, ctypes.c_float

NS_QUINTIC = (3.4445, -4.7750, 2.0315)
NS_CUBIC5 = ((3.3656576, -3.3420992), (2.5744352, -1.4957376), (2.5368962, -1.4312570),
             (2.4418906, -1.2764040), (2.2230472, -0.9630650))
PHASES_GRAM = (2, 3)
PHASES_DIRECT = (1, 1, 1, 1, 1)


# ------------------------------------------------------------------------------------ batched products
def _native_batched(a: torch.Tensor, b: torch.Tensor) -> bool:
    return (a.is_cuda and a.dtype == torch.bfloat16 and b.dtype == torch.bfloat16 and native.available()
            and a.shape[1] % 128 == 0 and a.shape[2] % 8 == 0 and b.shape[2] % 8 == 0)


def bmm_nt(a: torch.Tensor, b: torch.Tensor, b_mn: bool = False, alpha: float = 1.0, diag: float = 0.0) -> torch.Tensor:
    """Batched ``alpha * a[i] @ op(b[i]) + diag * I``: a (B, M, K); b (B, N, K) with ``b_mn`` false (product with b^T), or
    b (B, K, N) with ``b_mn`` true (plain product). One batched tcgen05 launch on a B200, ``torch.bmm`` elsewhere."""
    B, M, K = a.shape
    N = b.shape[2] if b_mn else b.shape[1]
    if not (_native_batched(a, b) and a.is_contiguous() and b.is_contiguous() and N % 8 == 0):
        out = torch.bmm(a, b if b_mn else b.transpose(1, 2))
        return affine(out, diag, alpha) if diag else (out if alpha == 1.0 else out * alpha)
    L = native.require()
    out = torch.empty(B, M, N, dtype=a.dtype, device=a.device)
    rc = L.kwu_gemm_bf16_batched(native.ptr(a), native.ptr(b), native.ptr(out), ci(B), ci(M), ci(N), ci(K), ci(int(b_mn)),
                                 cf(alpha), cf(diag), native.stream_ptr(), native.ptr(native.status_word()))
    native.check(rc, "muon batched gemm")
    return out


def _native_pass(x: torch.Tensor) -> bool:
    return x.is_cuda and x.dtype == torch.bfloat16 and native.available() and x.is_contiguous() and x.data_ptr() % 16 == 0


def affine(gram: torch.Tensor, a: float, b: float) -> torch.Tensor:
    """``a I + b G`` for a batch of square matrices, in one pass."""
    n = gram.shape[-1]
    if not (_native_pass(gram) and n % 8 == 0 and gram.numel()):
        return torch.add(torch.eye(n, dtype=gram.dtype, device=gram.device) * a, gram, alpha=b)
    L = native.require()
    out = torch.empty_like(gram)
    rc = L.kwu_diag_affine(native.ptr(gram), native.ptr(out), ci(gram.numel() // (n * n)), ci(n), cf(a), cf(b), native.stream_ptr())
    native.check(rc, "diag_affine")
    return out


def scale_transpose(x: torch.Tensor, norm: torch.Tensor | None, transpose: bool) -> torch.Tensor | None:
    """``x / norm`` (norm None: ``x``) of a bf16 (B, n, m) batch, transposed if asked, in one pass; None where the kernel
    does not apply."""
    B, R, C = x.shape
    if not (_native_pass(x) and R % 2 == 0 and C % 2 == 0 and x.numel() and B <= 65535 and R <= 65535 * 64):
        return None
    L = native.require()
    out = torch.empty((B, C, R) if transpose else (B, R, C), dtype=x.dtype, device=x.device)
    rc = L.kwu_scale_transpose(native.ptr(x), native.ptr(norm), native.ptr(out), ci(B), ci(R), ci(C), ci(int(transpose)),
                               native.stream_ptr())
    native.check(rc, "scale_transpose")
    return out


# ------------------------------------------------------------------------------------ Newton-Schulz
def _prepare(grad: torch.Tensor, dtype: torch.dtype):
    """(B, n, m) in ``dtype`` with n <= m and every matrix scaled to Frobenius norm 1 / 1.01; plus the flag that
    says the result must be transposed back."""
    x = grad.reshape(-1, grad.shape[-2], grad.shape[-1])
    norm = torch.linalg.vector_norm(x, dim=(-2, -1), keepdim=True, dtype=torch.float32).clamp_min(1e-7) * 1.01
    transposed = x.shape[-2] > x.shape[-1]
    if dtype == torch.bfloat16 and x.dtype == torch.bfloat16:
        done = scale_transpose(x, norm.reshape(-1), transposed)
        if done is not None:
            return done, transposed
    x = (x.float() / norm).to(dtype)
    if transposed:
        x = x.transpose(1, 2).contiguous()
    return x, transposed


def _finish(x: torch.Tensor, transposed: bool, shape) -> torch.Tensor:
    if transposed:
        done = scale_transpose(x, None, True)     # in place of a strided view, which the write-back would walk element by element
        x = x.transpose(1, 2) if done is None else done
    return x.reshape(shape)


def newton_schulz(grad: torch.Tensor, steps: int = 5, dtype: torch.dtype = torch.bfloat16,
                  coeffs=NS_QUINTIC) -> torch.Tensor:
    """Quintic iteration, batched over every leading dimension. Returns ``dtype``."""
    a, b, c = coeffs
    x, transposed = _prepare(grad, dtype)
    for _ in range(steps):
        gram = bmm_nt(x, x)                                   # X X^T
        poly = torch.add(gram * b, bmm_nt(gram, gram), alpha=c)   # b G + c G G (G is symmetric: G G^T = G G)
        x = torch.add(bmm_nt(poly, x, b_mn=True), x, alpha=a)
    return _finish(x, transposed, grad.shape)


def newton_schulz_cubic(grad: torch.Tensor, dtype: torch.dtype = torch.bfloat16, schedule=NS_CUBIC5,
                        phases=PHASES_DIRECT) -> torch.Tensor:
    """Cubic schedule with gram-space phases (see the module docstring). ``phases`` must sum to the number of
    steps of the schedule."""
    if sum(phases) != len(schedule):
        raise ValueError(f"phases {phases} sum to {sum(phases)}, the schedule has {len(schedule)} steps")
    x, transposed = _prepare(grad, dtype)
    k = 0
    for length in phases:
        product = step = gram = None
        for j in range(length):
            a, b = schedule[k + j]
            a = torch.tensor(a, dtype=x.dtype).item()         # the diagonal enters in the iteration's precision
            # G = X X^T, then S G S; S = a I + b G (symmetric). The last S of a phase is all that its G is for, so the
            # product that makes G writes S instead
            if j == 0:
                left, right, mn = x, x, False
            else:
                left, right, mn = bmm_nt(step, gram, b_mn=True), step, True
            if j + 1 == length:
                step = bmm_nt(left, right, b_mn=mn, alpha=b, diag=a)
            else:
                gram = bmm_nt(left, right, b_mn=mn)
                step = affine(gram, a, b)
            product = step if product is None else bmm_nt(step, product, b_mn=True)
        x = bmm_nt(product, x, b_mn=True)
        k += length
    return _finish(x, transposed, grad.shape)


def orthogonal_update_scale(shape, mode: str, rms_target: float = 0.2) -> float:
    rows, cols = shape[-2], shape[-1]
    if mode == "spectral":
        return max(1.0, rows / cols) ** 0.5
    if mode == "rms":
        return rms_target * max(rows, cols) ** 0.5
    raise ValueError(f"unknown update_scale {mode!r}; use 'spectral' or 'rms'")


# ------------------------------------------------------------------------------------ optimizer
class MuonW(torch.optim.Optimizer):
    """``hidden_params``: the matrices that take the orthogonalised step (>= 2-D; a stacked (E, out, in) expert
    weight is E matrices). ``adam_groups``: parameter groups for the internal AdamW (state in the parameter's
    dtype with the second moment stored as its square root, fp32 arithmetic)."""

    def __init__(self, hidden_params, adam_groups, lr: float = 3e-4, muon_lr: float = 0.02, weight_decay: float = 0.1,
                 betas=(0.9, 0.95), momentum: float = 0.95, nesterov: bool = True, ns_steps: int = 5,
                 ns_variant: str = "cubic5", ns_dtype: torch.dtype = torch.bfloat16, ns_batch_elems: int = 64 << 20,
                 gram_aspect: float = 1.5, update_scale: str = "spectral", rms_target: float = 0.2,
                 rounding: str = "nearest", seed: int = 0, eps: float = 1e-8, scale: str | None = None):
        if ns_variant not in ("cubic5", "quintic"):
            raise ValueError(f"unknown ns_variant {ns_variant!r}")
        if rounding not in ("nearest", "stochastic"):
            raise ValueError(f"unknown rounding rule {rounding!r}")
        update_scale = scale or update_scale
        hidden = list(hidden_params)
        for p in hidden:
            if p.dim() < 2:
                raise ValueError(f"a {p.dim()}-D parameter reached the Muon group: it has no singular values to equalise")
        # decay is decoupled and expressed per unit of the AdamW learning rate, so that both kinds of group
        # shrink at the same rate: wd_muon * muon_lr == weight_decay * lr
        groups = [{"params": hidden, "use_muon": True, "lr": muon_lr,
                   "weight_decay": weight_decay * lr / muon_lr if muon_lr else 0.0}]
        for g in adam_groups:
            if g["params"]:
                groups.append({"params": list(g["params"]), "use_muon": False, "lr": g.get("lr", lr),
                               "weight_decay": g.get("weight_decay", 0.0)})
        super().__init__(groups, dict(betas=betas, eps=eps))
        self.momentum, self.nesterov, self.ns_steps = momentum, nesterov, ns_steps
        self.ns_variant, self.ns_dtype, self.ns_batch_elems = ns_variant, ns_dtype, ns_batch_elems
        self.gram_aspect, self.update_scale, self.rms_target = gram_aspect, update_scale, rms_target
        self.stochastic, self.seed, self._sr_offset = rounding == "stochastic", seed, 0
        self._phases: dict[tuple, tuple] = {}

    # ------------------------------------------------------------------ helpers
    def phases_for(self, shape) -> tuple:
        """Gram-space grouping for wide shapes, direct steps for squarish ones (decided once per shape)."""
        key = tuple(shape[-2:])
        if key not in self._phases:
            short, long = sorted(key)
            self._phases[key] = PHASES_GRAM if long >= self.gram_aspect * short else PHASES_DIRECT
        return self._phases[key]

    def orthogonalize(self, batch: torch.Tensor) -> torch.Tensor:
        dtype = self.ns_dtype if batch.is_cuda else torch.float32
        if self.ns_variant == "cubic5":
            return newton_schulz_cubic(batch, dtype, phases=self.phases_for(batch.shape))
        return newton_schulz(batch, self.ns_steps, dtype)

    def _batch_size(self, shape) -> int:
        return max(1, self.ns_batch_elems // max(math.prod(shape), 1))

    # ------------------------------------------------------------------ step
    @torch.no_grad()
    def step(self, closure=None):
        loss = None
        if closure is not None:
            with torch.enable_grad():
                loss = closure()
        for group in self.param_groups:
            if group["use_muon"]:
                self._muon_group(group)
            else:
                self._adam_group(group)
        return loss

    def _muon_group(self, group) -> None:
        by_shape: dict[tuple, list] = {}
        for p in group["params"]:
            if p.grad is None:
                continue
            st = self.state[p]
            if "momentum_buffer" not in st:
                st["momentum_buffer"] = torch.zeros_like(p)
            by_shape.setdefault(tuple(p.shape), []).append(p)
        lr, wd, beta = group["lr"], group["weight_decay"], self.momentum
        for shape, params in by_shape.items():
            per = self._batch_size(shape)
            scale = orthogonal_update_scale(shape, self.update_scale, self.rms_target)
            for s in range(0, len(params), per):
                chunk = params[s:s + per]
                bufs = [self.state[p]["momentum_buffer"] for p in chunk]
                grads = [p.grad.to(b.dtype) for p, b in zip(chunk, bufs)]
                torch._foreach_lerp_(bufs, grads, 1 - beta)              # momentum EMA, one fused pass
                if self.nesterov:
                    direction = torch._foreach_lerp(grads, bufs, beta)   # look-ahead; .grad is left untouched
                else:
                    direction = bufs
                updates = self.orthogonalize(torch.stack(direction))    # (chunk, *shape)
                if self.stochastic and chunk[0].dtype == torch.bfloat16:
                    for p, u in zip(chunk, updates):
                        sr_update_(p, u.float().contiguous(), lr * wd, -lr * scale, seed=self.seed, offset=self._sr_offset)
                        self._sr_offset += p.numel()
                else:
                    torch._foreach_mul_(chunk, 1 - lr * wd)
                    torch._foreach_add_(chunk, [u.to(p.dtype) for p, u in zip(chunk, updates)], alpha=-lr * scale)

    def _adam_group(self, group) -> None:
        b1, b2 = group["betas"]
        for p in group["params"]:
            if p.grad is None:
                continue
            st = self.state[p]
            if "exp_avg" not in st:
                st["exp_avg"] = torch.zeros_like(p)
                st["exp_avg_rms"] = torch.zeros_like(p)
                st["step"] = 0
            st["step"] += 1
            adamw16_step_(p, st["exp_avg"], st["exp_avg_rms"], p.grad.to(p.dtype), lr=group["lr"], betas=(b1, b2),
                          eps=group["eps"], wd=group["weight_decay"], step=st["step"],
                          stochastic=self.stochastic and p.dtype == torch.bfloat16, seed=self.seed)
