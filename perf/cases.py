"""The work that is measured: what a training program has this package do, through its
public entry points, from the smallest calls to the largest.

Five kinds of case:

``adam``    one ``Adam.step()`` over the parameters of a Llama-shaped model whose
            gradients are there (the optimizer that keeps its state on the GPU).
``codec``   one weight through a packed format: ``copy_`` from a dense tensor (what an
            optimizer step and the load of a dense checkpoint do), ``dequantize``, or
            ``fake_quantize``.
``linear``  ``F.linear`` on a packed weight: forward only (evaluation, sampling) or
            forward and backward (training).
``eval``    the forward pass of a Llama-shaped model to its logits, without gradients.
``train``   a whole training step: forward and backward of ``accum`` micro-batches through
            the model and its chunked loss, and the step of ``Adam`` or ``OffloadAdam``,
            dense or with quantized linear layers.
"""

import math

import torch
import torch.nn.functional as F

from offload_adam_b200 import Adam, OffloadAdam
from offload_adam_b200.models.llama import LlamaConfig, build_llama
from offload_adam_b200.qweight import (Int4QWeight, Int8QWeight, NF4QWeight, NVFP4QWeight, fake_quantize,
                                       quantize_linears)

FORMATS = {"nvfp4": NVFP4QWeight, "nf4": NF4QWeight, "int4": Int4QWeight, "int8": Int8QWeight}
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
DTYPE_BYTES = {"bf16": 2, "fp16": 2, "fp32": 4}
# bytes of a packed weight element, block scales included
PACKED_BYTES = {"nvfp4": 0.5 + 1 / 16, "nf4": 0.5 + 4 / 64, "int4": 0.5 + 2 / 128, "int8": 1.0}
# bytes a step cannot do without, per element: gradient and moments in, moments and
# parameter out, plus the parameter in (where it is the source), the fp32 master or the
# int16 rounding error in and out
STEP_BYTES = {"stochastic_rounding": 14, "fp32_master": 20, "fp31_master": 18, "fp32_master_custom_rounding": 18}
MODES = tuple(STEP_BYTES)


def _dims(hidden, inter, layers, heads, kv_heads, vocab, tied=False):
    return dict(hidden=hidden, inter=inter, layers=layers, heads=heads, kv_heads=kv_heads, vocab=vocab, tied=tied)


TINY = _dims(256, 688, 2, 4, 4, 1024, tied=True)  # tiny_llama of models/llama.py


def wide(layers):
    """Layers of llama3_8b of models/llama.py, with its full vocabulary."""
    return _dims(4096, 14336, layers, 32, 8, 128256)


def listed():
    return [
        # the optimizer alone on a small model: 20 tensors, bound by launches and by the host
        dict(name="adam_tiny", kind="adam", mode="stochastic_rounding", **TINY),
        # a mid-size model with odd dimensions (tensor sizes that no vector width divides)
        dict(name="adam_odd", kind="adam", mode="fp31_master", **_dims(840, 2241, 1, 10, 5, 32003)),
        # one layer of the 8B shape with embedding and head, fp32 master: 1.3 G parameters
        dict(name="adam_wide", kind="adam", mode="fp32_master", **wide(1)),
        # re-quantization of one projection from its fp32 master
        dict(name="encode_nvfp4", kind="codec", op="quantize", format="nvfp4", dtype="fp32", rows=4096, cols=4096),
        # dense weights rounded to the int8 grid, ragged rows and columns
        dict(name="fake_int8_ragged", kind="codec", op="fake", format="int8", dtype="bf16", rows=4099, cols=1100),
        # sampling from a QAT model: one token through the largest projection of the 8B shape
        dict(name="linear_one_token_nf4", kind="linear", format="nf4", tokens=1, rows=14336, cols=4096,
             bias=False, backward=False),
        # a short ragged batch through a small projection with bias
        dict(name="linear_ragged_int4", kind="linear", format="int4", tokens=333, rows=2816, cols=1024,
             bias=True, backward=True),
        # QAT training, the usual 4096 tokens (2 x 2048)
        dict(name="linear_train_nvfp4", kind="linear", format="nvfp4", tokens=4096, rows=14336, cols=4096,
             bias=False, backward=True),
        # logits of a prompt
        dict(name="eval_wide", kind="eval", batch=1, seq=1024, **wide(2)),
        # the smallest training step: clipping, two micro-batches, offloaded matrices and
        # small tensors that stay on the GPU
        dict(name="train_tiny", kind="train", batch=2, seq=128, accum=2, optimizer="offload", mode="fp32_master",
             clip=True, quant="none", threshold=65536, **TINY),
        # QAT at the 8B shape: every linear layer but the head packed, state on the GPU
        dict(name="train_wide_int8", kind="train", batch=2, seq=2048, accum=1, optimizer="adam", mode="fp32_master",
             clip=False, quant="int8", threshold=1 << 20, **wide(2)),
        # the 8B shape with offloaded state, step inside backward, eight micro-batches of 4096
        dict(name="train_wide_offload", kind="train", batch=1, seq=4096, accum=8, optimizer="offload",
             mode="stochastic_rounding", clip=False, quant="none", threshold=1 << 20, **wide(4)),
    ]


# ---------------------------------------------------------------------------- draw
def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _odd_or_round(rng, lo, hi, to):
    """A size on a logarithmic scale: sometimes any number, more often a multiple of ``to``."""
    n = _log(rng, lo, hi)
    return max(1, int(n)) if rng.random() < 0.4 else max(to, int(n) // to * to)


def _draw_model(rng, max_hidden, max_params):
    while True:
        head_dim = rng.choice([32, 64, 64, 128, 128])
        heads = max(1, int(_log(rng, 2, max_hidden / head_dim + 0.99)))
        kv_heads = rng.choice([d for d in range(1, heads + 1) if heads % d == 0])
        hidden = heads * head_dim
        inter = max(64, int(hidden * rng.uniform(2.0, 4.0)) // 32 * 32)
        layers = rng.choice([1, 1, 2, 3, 4])
        vocab = _odd_or_round(rng, 1000, 128256, 64)
        tied = rng.random() < 0.4
        m = _dims(hidden, inter, layers, heads, kv_heads, vocab, tied)
        if sum(_params(m)) <= max_params:
            return m


def draw(rng):
    """One more case of the ranges above."""
    kind = rng.choice(["adam", "codec", "codec", "linear", "linear", "linear", "eval", "train", "train", "train"])
    if kind == "adam":
        while True:  # up to 64 outputs: parameters and state
            mode = rng.choice(MODES)
            m = _draw_model(rng, 4096, 1.2e9)
            if _n_tensors(m) * (3 if mode == "stochastic_rounding" else 4) <= 64:
                return dict(kind="adam", mode=mode, **m)
    if kind == "codec":
        op = rng.choice(["quantize", "quantize", "dequantize", "fake"])
        fmt = rng.choice(list(FORMATS))
        cols = int(_log(rng, 128, 16384)) // 128 * 128
        if fmt == "int8" and rng.random() < 0.4:
            cols = max(128, int(_log(rng, 128, 16384)) // 4 * 4)
        rows = _odd_or_round(rng, 64, min(32768, 2.0e8 / cols), 64)
        return dict(kind="codec", op=op, format=fmt, rows=rows, cols=cols,
                    dtype=rng.choice(["bf16", "fp32"] if op == "quantize" else ["bf16", "bf16", "fp16"]))
    if kind == "linear":
        backward = rng.random() < 0.5
        tokens = _odd_or_round(rng, 1, 8192, 8) if not backward else _odd_or_round(rng, 16, 8192, 64)
        cols = max(128, int(_log(rng, 256, 14336)) // 128 * 128)
        rows = max(128, int(_log(rng, 256, 14336)) // 32 * 32)
        return dict(kind="linear", format=rng.choice(list(FORMATS)), tokens=tokens, rows=rows, cols=cols,
                    bias=rng.random() < 0.25, backward=backward)
    while True:
        m = _draw_model(rng, 4096, 1.5e9)
        tokens = _log(rng, 64, 8192)
        batch = rng.choice([1, 1, 2, 4])
        seq = max(16, int(tokens / batch))
        if rng.random() < 0.7:
            seq = max(16, seq // 32 * 32)
        accum = rng.choice([1, 2, 4]) if kind == "train" else 1
        if 6 * sum(_params(m)) * batch * seq * accum > 1.0e14:
            continue
        if kind == "eval":
            return dict(kind="eval", batch=batch, seq=seq, **m)
        if _n_tensors(m) > 60:
            continue
        quant = rng.choice(["none", "none", "none"] + list(FORMATS))
        if m["hidden"] % 128 or m["inter"] % 128:  # the int4 group size
            quant = "none"
        mode = "fp32_master" if quant != "none" else rng.choice(MODES)
        optimizer = rng.choice(["adam", "offload", "offload"])
        if optimizer == "adam" and quant == "none" and rng.random() < 0.5:
            optimizer = "offload"
        # what goes back to the host per step must not be all that is measured
        if optimizer == "offload" and 1.4 * sum(_params(m)) * STEP_BYTES[mode] / 4 > 3e9:
            continue
        return dict(kind="train", batch=batch, seq=seq, accum=accum, optimizer=optimizer, mode=mode,
                    clip=optimizer == "offload" and rng.random() < 0.5, quant=quant, threshold=1 << 20, **m)


# ------------------------------------------------------------------------- prepare
def _config(c):
    return LlamaConfig(vocab_size=c["vocab"], hidden_size=c["hidden"], intermediate_size=c["inter"],
                       num_layers=c["layers"], num_heads=c["heads"], num_kv_heads=c["kv_heads"],
                       tie_embeddings=c["tied"])


def _layer_shapes(c):
    d = c["hidden"] // c["heads"]
    kv = c["kv_heads"] * d
    return [(c["hidden"], c["hidden"]), (kv, c["hidden"]), (kv, c["hidden"]), (c["hidden"], c["hidden"]),
            (c["inter"], c["hidden"]), (c["inter"], c["hidden"]), (c["hidden"], c["inter"])]


def _params(c):
    per_layer = [a * b for a, b in _layer_shapes(c)] + [c["hidden"]] * 2
    return per_layer * c["layers"] + [c["vocab"] * c["hidden"]] * (1 if c["tied"] else 2) + [c["hidden"]]


def _n_tensors(c):
    return len(_params(c))


class _Training:
    """What a training program holds: the model, its optimizer, the step's token ids."""

    def __init__(self, case, seed):
        gen = torch.Generator(device="cuda").manual_seed(seed)
        self.accum = case["accum"]
        self.model = build_llama(_config(case), device="cuda", seed=seed)
        self.model.train()
        if case["quant"] != "none":
            quantize_linears(self.model, FORMATS[case["quant"]], skip_patterns=("lm_head",))
        hp = dict(lr=1e-4, betas=(0.9, 0.999), eps=1e-8, weight_decay=0.01, mode=case["mode"],
                  decoupled_weight_decay=True, seed=seed)
        if case["optimizer"] == "adam":
            self.opt = Adam(self.model.parameters(), **hp)
        else:
            self.opt = OffloadAdam(self.model, max_grad_norm=1.0 if case["clip"] else None,
                                   inplace_param_threshold=case["threshold"], prefetch_policy="lazy", **hp)
        self.offload = case["optimizer"] == "offload"
        self.opt._quant_master_warned = True  # random weights: there is no checkpoint to refill from
        self.ids = [torch.randint(0, case["vocab"], (case["batch"], case["seq"]), device="cuda", generator=gen)
                    for _ in range(self.accum)]

    def __del__(self):
        if getattr(self, "offload", False):
            self.opt.close()  # finish what is in flight, take the hooks off the model


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]

    def normal(*shape, std=1.0, dtype=torch.bfloat16):
        return (torch.randn(shape, device="cuda", generator=gen) * std).to(dtype)

    if kind == "adam":
        model = build_llama(_config(case), device="cuda", seed=seed)
        for p in model.parameters():
            p.grad = torch.empty_like(p).normal_(std=1e-3, generator=gen)
        opt = Adam(model.parameters(), lr=1e-4, betas=(0.9, 0.999), eps=1e-8, weight_decay=0.01, mode=case["mode"],
                   decoupled_weight_decay=True, seed=seed)
        return dict(kind=kind, model=model, opt=opt)
    if kind == "codec":
        cls, dtype = FORMATS[case["format"]], DTYPES[case["dtype"]]
        x = normal(case["rows"], case["cols"], std=0.02, dtype=dtype)
        state = dict(kind=kind, op=case["op"], x=x, cls=cls)
        if case["op"] != "fake":
            outer = torch.bfloat16 if case["op"] == "quantize" else dtype
            kw = {"scale_dtype": outer} if case["format"] in ("int4", "int8") else {}
            state["q"] = cls.from_float(x.to(outer), **kw)
        return state
    if kind == "linear":
        cls = FORMATS[case["format"]]
        w = torch.nn.Parameter(cls.from_float(normal(case["rows"], case["cols"], std=0.02)))
        x = normal(case["tokens"], case["cols"])
        bias = torch.nn.Parameter(normal(case["rows"], std=0.02)) if case["bias"] else None
        state = dict(kind=kind, backward=case["backward"], w=w, x=x, bias=bias)
        if case["backward"]:
            x.requires_grad_(True)
            state["gy"] = normal(case["tokens"], case["rows"], std=1e-2)
        return state
    if kind == "eval":
        model = build_llama(_config(case), device="cuda", seed=seed).eval()
        ids = torch.randint(0, case["vocab"], (case["batch"], case["seq"]), device="cuda", generator=gen)
        return dict(kind=kind, model=model, ids=ids)
    return dict(kind=kind, training=_Training(case, seed))


# ----------------------------------------------------------------------------- run
def _plain(t):
    """A packed weight as its payload tensors, any other tensor as itself."""
    return t._payload() if hasattr(t, "_payload") else [t]


def run(state):
    kind = state["kind"]
    if kind == "adam":
        state["opt"].step()
        per_param = state["opt"].state
        return [[p.data] + [v for k, v in sorted(per_param[p].items()) if isinstance(v, torch.Tensor)]
                for p in state["model"].parameters()]
    if kind == "codec":
        if state["op"] == "quantize":
            state["q"].copy_(state["x"])
            return _plain(state["q"])
        if state["op"] == "dequantize":
            return state["q"].dequantize()
        return fake_quantize(state["x"], state["cls"])
    if kind == "linear":
        w, x, bias = state["w"], state["x"], state["bias"]
        if not state["backward"]:
            with torch.no_grad():
                return F.linear(x, w, bias)
        x.grad = w.grad = None
        if bias is not None:
            bias.grad = None
        y = F.linear(x, w, bias)
        y.backward(state["gy"])
        return [y.detach(), x.grad, w.grad] + ([] if bias is None else [bias.grad])
    if kind == "eval":
        with torch.no_grad():
            return state["model"](state["ids"])
    t = state["training"]
    for micro, ids in enumerate(t.ids):
        if t.offload:
            t.opt.ready_for_optimizer_step = micro == t.accum - 1
        loss = t.model(ids, labels=ids)
        (loss / t.accum).backward()
    t.opt.step()
    t.opt.zero_grad()
    return [loss.detach(), [_plain(p.data) for p in t.model.parameters()]]


# ---------------------------------------------------------------------------- work
def _forward_flops(c, logits=True):
    tokens = c["batch"] * c["seq"]
    linear = sum(a * b for a, b in _layer_shapes(c)) * c["layers"]
    attention = 2 * c["batch"] * c["seq"] ** 2 * c["hidden"] * c["layers"]  # causal: half of QK^T and PV
    return 2 * tokens * (linear + c["vocab"] * c["hidden"]) + attention


def work(case):
    kind = case["kind"]
    if kind == "adam":
        return {"bytes": sum(_params(case)) * STEP_BYTES[case["mode"]], "flops": 0}
    if kind == "codec":
        n = case["rows"] * case["cols"]
        dense, packed = DTYPE_BYTES[case["dtype"]], PACKED_BYTES[case["format"]]
        return {"bytes": n * (2 * dense if case["op"] == "fake" else dense + packed), "flops": 0}
    if kind == "linear":
        m, n, k = case["tokens"], case["rows"], case["cols"]
        moved, flops = n * k * PACKED_BYTES[case["format"]] + 2 * m * (n + k), 2 * m * n * k
        if case["backward"]:
            moved, flops = 2 * moved + 2 * n * k + 2 * m * k, 3 * flops
        return {"bytes": moved, "flops": flops}
    n = sum(_params(case))
    tokens = case["batch"] * case["seq"]
    if kind == "eval":
        return {"bytes": 2 * n + 2 * tokens * case["vocab"], "flops": _forward_flops(case)}
    # forward and backward read the weights once each and write their gradients once
    return {"bytes": n * (6 * case["accum"] + STEP_BYTES[case["mode"]]), "flops": 3 * case["accum"] * _forward_flops(case)}


# ----------------------------------------------------------------------- tolerance
def tolerance(case):
    kind = case["kind"]
    if kind in ("adam", "codec"):
        return "exact"  # every operation of the step and of the formats has a defined rounding
    if kind == "linear":
        return {"rel": 8e-3}  # bf16 results against fp64: 1.7e-3 to 2.4e-3
    if kind == "eval":
        # elementwise parts and attention in fp32 against bf16 steps, one to three layers: 0.5e-2 to 1.7e-2
        return {"rel": 3e-2}
    # the same comparison after one and two steps: 0.4e-3 to 1.7e-3 of the weights (rounding
    # flips the sign of updates whose gradient is near zero); the updates themselves are 5e-3
    return {"rel": 3e-3, "differ": 1e-2}
