"""Self-contained Llama-style causal LM used by the examples and benchmarks.

The reference's examples train a HuggingFace ``AutoModelForCausalLM`` with SDPA
attention, gradient checkpointing and a fused linear cross-entropy
(reference: examples/e2e_train/train.py:106-129).  This module provides the same
ingredients without external model code: RMSNorm, rotary embeddings, grouped
query attention through ``scaled_dot_product_attention``, SwiGLU, optional
per-layer activation checkpointing and a chunked linear + cross-entropy head
that holds the logits of a few thousand tokens at most, in bf16.

Parameter names and shapes match the HF Llama layout (``model.embed_tokens``,
``model.layers.N.self_attn.{q,k,v,o}_proj``, ``mlp.{gate,up,down}_proj``,
``input_layernorm``, ``post_attention_layernorm``, ``model.norm``, ``lm_head``)
so checkpoints and the quantization name filters line up.
"""

from __future__ import annotations

from dataclasses import dataclass
from typing import Optional

import torch
import torch.nn as nn
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

from .. import _ext
from ..ops.dispatch import use_kernels


@dataclass
class LlamaConfig:
    vocab_size: int = 128256
    hidden_size: int = 4096
    intermediate_size: int = 14336
    num_layers: int = 32
    num_heads: int = 32
    num_kv_heads: int = 8
    rope_theta: float = 500000.0
    rms_eps: float = 1e-5
    tie_embeddings: bool = False
    init_std: float = 0.02
    ce_chunk: int = 2048  # rows of the logits that the loss head holds (see _CE_ROWS_PER_CHUNK)
    head_dim_override: Optional[int] = None  # Qwen3: 128 whatever hidden_size / num_heads is
    qk_norm: bool = False  # Qwen3: RMSNorm over head_dim on queries and keys before RoPE

    @property
    def head_dim(self):
        return self.head_dim_override or self.hidden_size // self.num_heads


def llama3_8b(**kw) -> LlamaConfig:
    return LlamaConfig(**kw)


def llama3_70b(**kw) -> LlamaConfig:
    base = dict(hidden_size=8192, intermediate_size=28672, num_layers=80, num_heads=64, num_kv_heads=8)
    base.update(kw)
    return LlamaConfig(**base)


def qwen3_8b(**kw) -> LlamaConfig:
    """Qwen3-8B shape, the model of the reference's published tables (reference:
    examples/e2e_train/README.md:36-54): 36 layers, hidden 4096, 32 query / 8 KV heads
    of 128, SwiGLU 12288, vocabulary 151936, RoPE theta 1e6, RMSNorm on q and k."""
    base = dict(vocab_size=151936, hidden_size=4096, intermediate_size=12288, num_layers=36, num_heads=32,
                num_kv_heads=8, rope_theta=1e6, rms_eps=1e-6, head_dim_override=128, qk_norm=True)
    base.update(kw)
    return LlamaConfig(**base)


def tiny_llama(**kw) -> LlamaConfig:
    """2 layers, hidden 256, 4 heads, SwiGLU 688, vocab 1024, tied embeddings."""
    base = dict(vocab_size=1024, hidden_size=256, intermediate_size=688, num_layers=2, num_heads=4,
                num_kv_heads=4, rope_theta=1e4, tie_embeddings=True, ce_chunk=128)
    base.update(kw)
    return LlamaConfig(**base)


class RMSNorm(nn.Module):
    def __init__(self, dim, eps):
        super().__init__()
        self.weight = nn.Parameter(torch.ones(dim))
        self.eps = eps

    def _kernel_takes(self, *xs):
        # shorter rows (q_norm / k_norm) would leave most of a warp idle
        w, cols = self.weight, self.weight.shape[0]
        return (use_kernels(w, *xs) and 256 <= cols <= _ext.load(required=True).NORM_MAX_COLS and cols % 8 == 0
                and all(x.numel() > 0 and x.shape[-1] == cols and x.device == w.device for x in xs))

    def forward(self, x):
        if not torch.jit.is_scripting():
            if self._kernel_takes(x):
                return _ext.load(required=True).rms_norm(x, self.weight, self.eps)
        return F.rms_norm(x, (x.shape[-1],), self.weight, self.eps)


_FORWARD = {cls: cls.forward for cls in (RMSNorm, nn.Embedding)}


def _bare_call(module):
    """True when calling ``module`` runs its class's own ``forward`` and nothing else: no hook,
    no ``forward`` put in its place on the instance or on the class, no compiled call."""
    return not (module._forward_hooks or module._forward_pre_hooks or module._backward_hooks
                or module._backward_pre_hooks or nn.modules.module._has_any_global_hook()
                or "forward" in module.__dict__ or type(module).forward is not _FORWARD[type(module)]
                or module._compiled_call_impl is not None)


def _add_norm(x, delta, norm):
    """``(x + delta, norm(x + delta))``, in one kernel unless somebody watches or replaces the
    module's calls."""
    if type(norm) is RMSNorm and norm._kernel_takes(x, delta) and x.shape == delta.shape and _bare_call(norm):
        return _ext.load(required=True).add_rms_norm(x, delta, norm.weight, norm.eps)
    x = x + delta
    return x, norm(x)


def _rope_tables(seq_len, head_dim, theta, device):
    inv = 1.0 / (theta ** (torch.arange(0, head_dim, 2, device=device, dtype=torch.float32) / head_dim))
    t = torch.arange(seq_len, device=device, dtype=torch.float32)
    ang = torch.outer(t, inv)
    ang = torch.cat([ang, ang], dim=-1)
    return ang.cos(), ang.sin()


def _apply_rope(x, cos, sin):
    # x: (B, H, S, D); rotate-half convention
    d = x.shape[-1] // 2
    rot = torch.cat([-x[..., d:], x[..., :d]], dim=-1)
    return x * cos + rot * sin


def _rope_heads(q, k, cos, sin, hd):
    """Rotated ``(batch, seq, heads, hd)`` queries and keys, as ``(batch, heads, seq, hd)``."""
    # heads in whole pairs of 8-value vectors, tables as _rope_for makes them
    if (hd % 16 == 0 and use_kernels(q, k, cos, sin) and cos.shape == sin.shape == (q.shape[1], hd)
            and cos.is_contiguous() and sin.is_contiguous() and not (cos.requires_grad or sin.requires_grad)
            and q.device == k.device == cos.device == sin.device):
        q, k = _ext.load(required=True).rope(q, k, cos, sin)
        return q.transpose(1, 2), k.transpose(1, 2)
    return _apply_rope(q.transpose(1, 2), cos, sin), _apply_rope(k.transpose(1, 2), cos, sin)


def _embed(module, ids):
    """``module(ids)``; a training step's dense gradient of the table comes from one kernel
    that also writes the zero rows.  Plain ``nn.Embedding`` without options, nobody watching."""
    if type(module) is nn.Embedding:
        w = module.weight
        if (w.requires_grad and torch.is_grad_enabled() and use_kernels(w) and w.shape[1] % 8 == 0
                and module.padding_idx is None and module.max_norm is None
                and not (module.scale_grad_by_freq or module.sparse)
                and type(ids) is torch.Tensor and ids.dtype == torch.int64 and ids.device == w.device
                and _ext.load(required=True).embed_kernel_wins(ids.numel(), *w.shape) and _bare_call(module)):
            return _ext.load(required=True).embedding(w, ids)
    return module(ids)


class Attention(nn.Module):
    def __init__(self, cfg: LlamaConfig):
        super().__init__()
        h, d = cfg.hidden_size, cfg.head_dim
        self.nh, self.nkv, self.hd = cfg.num_heads, cfg.num_kv_heads, d
        self.q_proj = nn.Linear(h, self.nh * d, bias=False)
        self.k_proj = nn.Linear(h, self.nkv * d, bias=False)
        self.v_proj = nn.Linear(h, self.nkv * d, bias=False)
        self.o_proj = nn.Linear(self.nh * d, h, bias=False)
        if cfg.qk_norm:  # parameter names as in HF Qwen3: self_attn.q_norm / k_norm
            self.q_norm = RMSNorm(d, cfg.rms_eps)
            self.k_norm = RMSNorm(d, cfg.rms_eps)
        else:
            self.q_norm = self.k_norm = None

    def forward(self, x, cos, sin):
        B, S, _ = x.shape
        q = self.q_proj(x).view(B, S, self.nh, self.hd)
        k = self.k_proj(x).view(B, S, self.nkv, self.hd)
        if self.q_norm is not None:
            q, k = self.q_norm(q), self.k_norm(k)
        v = self.v_proj(x).view(B, S, self.nkv, self.hd).transpose(1, 2)
        if torch.jit.is_scripting():
            q = _apply_rope(q.transpose(1, 2), cos, sin)
            k = _apply_rope(k.transpose(1, 2), cos, sin)
        else:
            q, k = _rope_heads(q, k, cos, sin, self.hd)
        o = F.scaled_dot_product_attention(q, k, v, is_causal=True, enable_gqa=self.nh != self.nkv)
        return self.o_proj(o.transpose(1, 2).reshape(B, S, self.nh * self.hd))


class MLP(nn.Module):
    def __init__(self, cfg: LlamaConfig):
        super().__init__()
        self.gate_proj = nn.Linear(cfg.hidden_size, cfg.intermediate_size, bias=False)
        self.up_proj = nn.Linear(cfg.hidden_size, cfg.intermediate_size, bias=False)
        self.down_proj = nn.Linear(cfg.intermediate_size, cfg.hidden_size, bias=False)

    def forward(self, x):
        gate, up = self.gate_proj(x), self.up_proj(x)
        if not torch.jit.is_scripting():
            if use_kernels(gate, up) and gate.shape == up.shape and gate.device == up.device:
                return self.down_proj(_ext.load(required=True).swiglu(gate, up))
        return self.down_proj(F.silu(gate) * up)


class DecoderLayer(nn.Module):
    def __init__(self, cfg: LlamaConfig):
        super().__init__()
        self.input_layernorm = RMSNorm(cfg.hidden_size, cfg.rms_eps)
        self.self_attn = Attention(cfg)
        self.post_attention_layernorm = RMSNorm(cfg.hidden_size, cfg.rms_eps)
        self.mlp = MLP(cfg)

    def forward(self, x, cos, sin):
        attn = self.self_attn(self.input_layernorm(x), cos, sin)
        if torch.jit.is_scripting():
            x = x + attn
            h = self.post_attention_layernorm(x)
        else:
            x, h = _add_norm(x, attn, self.post_attention_layernorm)
        return x + self.mlp(h)


class _ChunkedLinearCE(torch.autograd.Function):
    """mean cross-entropy of ``h @ W^T`` against ``labels`` (ignore_index=-100), in the
    operations of PyTorch, chunk by chunk.  Gradients with respect to ``h`` and ``W`` are
    formed in the same pass and only scaled in backward, so the logits of a chunk are live
    for one chunk only."""

    @staticmethod
    def forward(ctx, h, weight, labels, chunk):
        N, H = h.shape
        valid = labels != -100
        n_valid = valid.sum().clamp(min=1)
        loss = torch.zeros((), dtype=torch.float32, device=h.device)
        gh = torch.empty_like(h)
        gw = torch.zeros(weight.shape, dtype=torch.float32, device=h.device)
        inv = 1.0 / n_valid.float()
        for s in range(0, N, chunk):
            e = min(N, s + chunk)
            logits = (h[s:e] @ weight.T).float()
            lab = labels[s:e]
            lse = torch.logsumexp(logits, dim=-1)
            msk = valid[s:e]
            safe = lab.clamp(min=0)
            picked = logits.gather(1, safe[:, None]).squeeze(1)
            loss += ((lse - picked) * msk).sum()
            probs = torch.softmax(logits, dim=-1)
            probs.scatter_add_(1, safe[:, None], -torch.ones_like(picked)[:, None])
            probs *= (msk.float() * inv)[:, None]
            d = probs.to(h.dtype)
            gh[s:e] = d @ weight
            gw.add_(d.T @ h[s:e])
        ctx.save_for_backward(gh, gw.to(weight.dtype))
        return loss * inv

    @staticmethod
    def backward(ctx, g):
        gh, gw = ctx.saved_tensors
        return gh * g.to(gh.dtype), gw * g.to(gw.dtype), None, None


# Rows of the logits that the kernel route handles at a time, in units of the caller's chunk.
# With c rows a chunk, V words and hidden size H, the PyTorch route's peak is the larger of
# 16 c V + 4 V H bytes (two chunks' logits in fp32 and bf16, the fp32 gradient of the head) and
# 10 c V + 6 V H (one chunk, and a product that is added).  Here one group of R rows takes
# 4 R V + 2 V H (bf16 logits and their gradient, the gradient of the head), several groups
# 2 R V + 6 V H: R = 4 c stays below it for every H.  Measured for 4096 rows, c = 2048, hidden
# 1024, 128256 words: 2.2 GB, PyTorch route 4.7; 20000 rows, hidden 256, 32000 words: 0.6 and 1.1.
_CE_ROWS_PER_CHUNK = 4


def _head_logits(h, weight, out, chunk):
    """``out = h @ weight.T``.  A vocabulary that is no multiple of 8 takes the library's
    kernels for unaligned operands, which may split a sum and add its parts in bf16; how many
    rows there are decides it.  Those take the caller's chunk (840 x 32003: 0.17 % off 64 bits
    for 2048 rows at a time, 0.20 % for 8192)."""
    if weight.shape[0] % 8 == 0 or h.shape[0] <= chunk:
        torch.mm(h, weight.T, out=out)
        return
    for s in range(0, h.shape[0], chunk):
        torch.mm(h[s:s + chunk], weight.T, out=out[s:s + chunk])


def _hidden_grad(d, weight, rows, out=None):
    """``d @ weight``.  For the same vocabularies the sum over the words is kept in fp32
    to its end, ``rows`` rows at a time: split sums in bf16 left 0.2 to 1 % of error (60 rows of
    32003 words, hidden 64: 0.57 %), fp32 leaves the 0.17 % of the one rounding, in the same
    time (32003 x 840, 8192 rows: 3656 us, 3645 in bf16)."""
    if d.shape[1] % 8 == 0:
        return torch.mm(d, weight, out=out)
    if out is None:
        out = torch.empty((d.shape[0], weight.shape[1]), dtype=d.dtype, device=d.device)
    for s in range(0, d.shape[0], rows):
        out[s:s + rows] = torch.mm(d[s:s + rows], weight, out_dtype=torch.float32)
    return out


class _KernelLinearCE(torch.autograd.Function):
    """The same loss through ``csrc/loss_ops.cu`` (bf16, CUDA).

    Up to ``_CE_ROWS_PER_CHUNK`` chunks of rows: forward keeps the bf16 logits and two floats
    a row; backward turns them into the gradient of the logits, the incoming gradient
    folded in, and both matrix products run once over all rows, accumulating in fp32.
    More rows than that: gradients are formed in forward, a group of rows at a time, and
    scaled in backward."""

    @staticmethod
    def forward(ctx, h, weight, labels, chunk):
        C = _ext.load(required=True)
        N, V = h.shape[0], weight.shape[0]
        f32 = dict(dtype=torch.float32, device=h.device)
        loss, inv = torch.empty((), **f32), torch.empty((), **f32)
        ctx.want_grad = ctx.needs_input_grad[0] or ctx.needs_input_grad[1]
        rows = chunk * _CE_ROWS_PER_CHUNK
        ctx.one_group = N <= rows
        logits = C.ce_logits_buffer(h, min(N, rows), V)
        stats = torch.empty(3 * logits.shape[0], **f32)
        if ctx.one_group:
            _head_logits(h, weight, logits, chunk)
            C.ce_stats(logits, labels, stats)
            C.ce_finish(stats[2 * N:], labels, loss, inv)
            if ctx.want_grad:
                ctx.save_for_backward(h, weight, labels, logits, stats, inv)
            return loss
        row_loss = torch.empty(N, **f32)
        if ctx.want_grad:
            C.ce_finish(None, labels, None, inv)
            gh = torch.empty_like(h)
            gw = None
        for s in range(0, N, rows):
            n = min(N - s, rows)
            hs, lab, lo, st = h[s:s + n], labels[s:s + n], logits[:n], stats[:3 * n]
            _head_logits(hs, weight, lo, chunk)
            C.ce_stats(lo, lab, st)
            row_loss[s:s + n] = st[2 * n:]
            if ctx.want_grad:
                C.ce_grad(lo, lab, st, inv, None, lo)
                _hidden_grad(lo, weight, max(V // 2, 128), gh[s:s + n])
                if gw is None:  # fp32 until the last; two groups are one sum
                    gw = lo.T @ hs if N <= 2 * rows else torch.mm(lo.T, hs, out_dtype=torch.float32)
                else:
                    part = lo.T @ hs
                    gw = C.sum_bf16(gw, part, s + rows >= N, part)
                    del part  # or it lives beside the next one
        C.ce_finish(row_loss, labels, loss, inv)
        if ctx.want_grad:
            ctx.save_for_backward(gh, gw)
        return loss

    @staticmethod
    def backward(ctx, g):
        if not ctx.one_group:
            gh, gw = ctx.saved_tensors
            return gh * g.to(gh.dtype), gw * g.to(gw.dtype), None, None
        C = _ext.load(required=True)
        h, weight, labels, logits, stats, inv = ctx.saved_tensors
        V = weight.shape[0]
        through = g.requires_grad and torch.is_grad_enabled()  # keep the graph through g
        # saved-tensor hooks may have returned copies without the padded rows
        if logits.stride(0) % 16 or logits.data_ptr() % 32 or not _whole_vectors(logits):
            logits = C.ce_logits_buffer(logits, *logits.shape).copy_(logits)
        d = C.ce_logits_buffer(logits, *logits.shape)
        with torch.no_grad():
            C.ce_grad(logits, labels, stats, inv, None if through else g.detach().float().contiguous(), d)
            gh = gw = None
            if ctx.needs_input_grad[0]:
                gh = _hidden_grad(d, weight, max(V, 128))
            if ctx.needs_input_grad[1]:
                gw = d.T @ h
        if through:
            gh = None if gh is None else gh * g.to(gh.dtype)
            gw = None if gw is None else gw * g.to(gw.dtype)
        return gh, gw, None, None


def _whole_vectors(x):
    """True when every row of the 2-D view ``x``, the last one too, can be read up to the
    next multiple of 16 elements without leaving the storage."""
    end = x.storage_offset() + (x.shape[0] - 1) * x.stride(0) + (x.shape[1] + 15) // 16 * 16
    return x.stride(1) == 1 and end * x.element_size() <= x.untyped_storage().nbytes()


def chunked_linear_cross_entropy(h, weight, labels, chunk=2048):
    kernels = (use_kernels(h, weight) and h.dim() == 2 and weight.dim() == 2 and h.numel() > 0 and weight.numel() > 0
               and h.shape[1] % 8 == 0  # all operands of the products would be unaligned
               and type(labels) is torch.Tensor and labels.is_cuda and labels.dtype == torch.int64
               and labels.shape == h.shape[:1] and h.device == weight.device == labels.device)
    if kernels:
        return _KernelLinearCE.apply(h, weight, labels.contiguous(), chunk)
    return _ChunkedLinearCE.apply(h, weight, labels, chunk)


class LlamaModel(nn.Module):
    def __init__(self, cfg: LlamaConfig):
        super().__init__()
        self.embed_tokens = nn.Embedding(cfg.vocab_size, cfg.hidden_size)
        self.layers = nn.ModuleList([DecoderLayer(cfg) for _ in range(cfg.num_layers)])
        self.norm = RMSNorm(cfg.hidden_size, cfg.rms_eps)


class LlamaForCausalLM(nn.Module):
    def __init__(self, cfg: LlamaConfig):
        super().__init__()
        self.config = cfg
        self.model = LlamaModel(cfg)
        self.lm_head = nn.Linear(cfg.hidden_size, cfg.vocab_size, bias=False)
        if cfg.tie_embeddings:
            self.lm_head.weight = self.model.embed_tokens.weight
        self.gradient_checkpointing = False
        self._rope = None
        self.reset_parameters()

    def reset_parameters(self):
        std = self.config.init_std
        for m in self.modules():
            if isinstance(m, (nn.Linear, nn.Embedding)):
                nn.init.normal_(m.weight, mean=0.0, std=std)

    def gradient_checkpointing_enable(self):
        self.gradient_checkpointing = True

    def gradient_checkpointing_disable(self):
        self.gradient_checkpointing = False

    def _rope_for(self, S, device, dtype):
        key = (S, device, dtype)
        if self._rope is None or self._rope[0] != key:
            cos, sin = _rope_tables(S, self.config.head_dim, self.config.rope_theta, device)
            self._rope = (key, cos.to(dtype), sin.to(dtype))
        return self._rope[1], self._rope[2]

    def hidden_states(self, input_ids):
        x = _embed(self.model.embed_tokens, input_ids)
        cos, sin = self._rope_for(input_ids.shape[1], x.device, x.dtype)
        for layer in self.model.layers:
            if self.gradient_checkpointing and self.training:
                x = checkpoint(layer, x, cos, sin, use_reentrant=False)
            else:
                x = layer(x, cos, sin)
        return self.model.norm(x)

    def forward(self, input_ids, labels: Optional[torch.Tensor] = None):
        """Returns the mean next-token loss when ``labels`` is given (labels are
        shifted here, as in HF models), else the full logits."""
        h = self.hidden_states(input_ids)
        if labels is None:
            return self.lm_head(h)
        B, S, H = h.shape
        shift = torch.full_like(labels, -100)
        shift[:, :-1] = labels[:, 1:]
        return chunked_linear_cross_entropy(h.reshape(B * S, H), self.lm_head.weight,
                                            shift.reshape(-1), self.config.ce_chunk)


def build_llama(cfg: LlamaConfig, device="cuda", dtype=torch.bfloat16, seed=0, symmetric_group=None,
                symmetric_threshold=1024 * 1024) -> LlamaForCausalLM:
    """Random-init model (N(0, init_std), norms at 1) created directly on ``device`` and
    directly in ``dtype``: no fp32 copy of the weights ever exists (a 70B model would not
    fit otherwise).  With ``symmetric_group`` (a process group) the large parameters are
    created in symmetric memory, where the peer-memory path of ``DistributedOffloadAdam``
    wants them, so that no second copy of the weights is needed when the optimizer is
    built (``parallel.symm.materialize_in_symmetric_memory``)."""
    gen_state = torch.random.get_rng_state()
    default_dtype = torch.get_default_dtype()
    torch.manual_seed(seed)
    try:
        torch.set_default_dtype(dtype)
        if symmetric_group is None:
            with torch.device(device):
                model = LlamaForCausalLM(cfg)
            model = model.to(dtype)
        else:
            from ..parallel.symm import materialize_in_symmetric_memory
            with torch.device("meta"):
                model = LlamaForCausalLM(cfg)
            materialize_in_symmetric_memory(model, device, symmetric_group, symmetric_threshold, dtype)
            with torch.no_grad():
                for p in model.parameters():
                    if p.dim() == 1:
                        p.fill_(1.0)  # norm weights
                model.reset_parameters()
    finally:
        torch.set_default_dtype(default_dtype)
        torch.random.set_rng_state(gen_state)
    return model
