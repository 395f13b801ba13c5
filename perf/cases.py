"""The work that a program using this package has it do, as measured cases.

``listed()`` names them, ``draw(rng)`` gives more of the same ranges, ``prepare`` builds what such a program holds before
the call, ``run`` is one pass through the public entry points, ``work`` what a pass cannot do without and ``tolerance``
how far another correct implementation at the same precision may be off.

Kinds:

``step``       one optimizer step: forward, chunked linear + cross-entropy, backward, clip to norm 1, AdamW.  With
               ``ddp`` the loop is the Trainer's (gradient buckets, device-resident clip coefficient, bf16 shadows written
               by the optimizer), without it the plain loop of a script (autograd gradients, ``clip_grad_norm``).
``eval``       held-out loss without gradients, padded targets among the labels.
``logits``     forward of a prompt to logits.
``linear_ce``  the fused linear + cross-entropy alone, forward and backward.
``attention``  the differentiable attention op on its own q / k / v tensors, forward and backward.
``optimizer``  clip + AdamW over a parameter list.
"""

from __future__ import annotations

import math

import torch

from torchure_b200.core.grad_helper import clip_grad_norm
from torchure_b200.loss import fused_linear_cross_entropy, shift_labels
from torchure_b200.models import build_model
from torchure_b200.objectives import build_objective
from torchure_b200.ops.attention import flash_attention
from torchure_b200.optim import build_optimizer
from torchure_b200.parallel.ddp import DDP

IGNORE = -100
ADAMW = {"lr": 3e-4, "weight_decay": 0.1, "betas": [0.9, 0.95], "fused": True}     # the shipped configurations

QWEN3_06B = dict(layers=28, heads=16, kv_heads=8, emb=1024, ffn=3072, vocab=151936, qk_norm=True)
QWEN3_4B = dict(heads=32, kv_heads=8, emb=2560, ffn=9728, vocab=151936, qk_norm=True)
LLAMA3_1B = dict(layers=16, heads=16, kv_heads=4, emb=2048, ffn=8192, vocab=128256, qk_norm=False)


class Program(dict):
    """State of a training program.  One that ends hands its gradient hooks back: the parameters and the bucket reducer
    hold on to each other through them, and a process that builds several models would keep every one."""

    def __del__(self):
        for p in self.get("params", ()):
            hooks = getattr(p, "_post_accumulate_grad_hooks", None)
            if hooks:
                hooks.clear()


class OneRank:
    """Mesh of one rank: what a single-GPU program hands to the data-parallel wrapper and to ``clip_grad_norm``."""

    def size(self, dim):
        return 1

    def coordinate(self, dim):
        return 0

    def get_group(self, dim):
        return None


def listed():
    return [
        # the smallest training step (a smoke run, a unit test, a first try on a laptop-sized model): launches and latency
        dict(name="step_tiny", kind="step", ddp=False, layers=2, heads=4, kv_heads=2, emb=512, ffn=1024, vocab=8192,
             qk_norm=True, batch=2, seq=512, micro=1, chunk=512),
        # the headline configuration: Qwen3-0.6B, two packed sequences of 4096 tokens per GPU
        dict(name="step_qwen3_0.6b", kind="step", ddp=True, batch=2, seq=4096, micro=1, chunk=4096, **QWEN3_06B),
        # the same width, shallower, with gradient accumulation over two micro-batches of an odd number of 128-token blocks
        dict(QWEN3_06B, name="step_accumulate", kind="step", ddp=True, layers=6, batch=3, seq=1408, micro=2, chunk=4096),
        # the shipped Llama 3.2 1B configuration: no QK-norm, four query heads per KV head, hidden 2048
        dict(name="step_llama3_1b", kind="step", ddp=True, batch=2, seq=4096, micro=1, chunk=4096, **LLAMA3_1B),
        # blocks and head of the 4B configuration at its batch of one sequence (a pipeline or test cut of the depth)
        dict(QWEN3_4B, name="step_qwen3_4b_cut", kind="step", ddp=True, layers=4, batch=1, seq=4096, micro=1, chunk=4096),
        # held-out evaluation of the 0.6B model
        dict(name="eval_qwen3_0.6b", kind="eval", batch=4, seq=2048, chunk=4096, ignored=0.1, **QWEN3_06B),
        # scoring one short prompt: the smallest forward the kernels take
        dict(name="logits_short", kind="logits", batch=1, seq=128, **QWEN3_06B),
        # the loss head alone at the benchmark's size, bf16 weight
        dict(name="linear_ce_8k", kind="linear_ce", rows=8192, dim=1024, vocab=151936, chunk=4096, ignored=0.0, weight="bf16"),
        # ... and ragged: a vocabulary and a row count that fill no tile, fp32 weight, padded targets
        dict(name="linear_ce_ragged", kind="linear_ce", rows=1531, dim=512, vocab=50257, chunk=600, ignored=0.1,
             weight="fp32"),
        # long context: one sequence of 16k tokens
        dict(name="attention_16k", kind="attention", batch=1, seq=16384, kv_seq=16384, heads=16, kv_heads=8, causal=True),
        # an off-diagonal block pair: every query sees every key, unequal lengths
        dict(name="attention_pair", kind="attention", batch=2, seq=384, kv_seq=896, heads=8, kv_heads=2, causal=False),
        # clip + AdamW over the tensors of four 4B blocks and a vocabulary cut, odd sizes among them
        dict(name="optimizer", kind="optimizer", blocks=4, heads=32, kv_heads=8, emb=2560, ffn=9728, vocab=32001),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _model_dims(rng):
    kv = rng.choice([1, 2, 3, 4, 6, 8])
    emb = 128 * int(_log(rng, 2, 20.99))
    return dict(layers=int(_log(rng, 1, 16.99)), heads=kv * rng.choice([2, 4]), kv_heads=kv, emb=emb,
                ffn=64 * int(emb * rng.uniform(2, 4) / 64), vocab=8 * int(_log(rng, 512, 18992)),
                qk_norm=rng.random() < 0.7)


def draw(rng):
    kind = rng.choice(["step", "step", "step", "eval", "logits", "linear_ce", "attention", "optimizer"])
    if kind in ("step", "eval", "logits"):
        d = _model_dims(rng)
        if kind == "logits":
            return dict(kind=kind, batch=rng.randint(1, 4), seq=128 * int(_log(rng, 1, 8.99)), **d)
        seq = 128 * int(_log(rng, 1, 32.99))
        batch = rng.randint(1, max(1, min(8, 8192 // seq)))
        chunk = rng.choice([512, 1000, 1024, 4096])
        if kind == "eval":
            return dict(kind=kind, batch=batch, seq=seq, chunk=chunk, ignored=rng.choice([0.0, 0.1, 0.3]), **d)
        micro = 2 if batch * seq <= 4096 and rng.random() < 0.3 else 1
        # without the wrapper every parameter's gradient is a tensor of its own: shallow models
        ddp = d["layers"] > 4 or rng.random() < 0.6
        return dict(kind=kind, ddp=ddp, batch=batch, seq=seq, micro=micro if ddp else 1, chunk=chunk, **d)
    if kind == "linear_ce":
        return dict(kind=kind, rows=int(_log(rng, 100, 8192)), dim=64 * int(_log(rng, 4, 32.99)),
                    vocab=int(_log(rng, 4000, 151936)), chunk=rng.choice([512, 1000, 1024, 4096]),
                    ignored=rng.choice([0.0, 0.1]), weight=rng.choice(["bf16", "fp32"]))
    if kind == "attention":
        kv = rng.choice([1, 2, 3, 4, 8])
        heads = kv * rng.choice([2, 4])
        seq = 128 * int(_log(rng, 1, 64.99))
        causal = rng.random() < 0.6
        kv_seq = seq if causal else 128 * int(_log(rng, 1, 64.99))
        return dict(kind=kind, batch=rng.randint(1, max(1, min(4, 16384 // max(seq, kv_seq)))), seq=seq, kv_seq=kv_seq,
                    heads=heads, kv_heads=kv, causal=causal)
    kv = rng.choice([2, 4, 8])
    emb = int(_log(rng, 256, 2560))
    return dict(kind=kind, blocks=rng.randint(1, 4), heads=kv * 2, kv_heads=kv, emb=emb, ffn=int(emb * rng.uniform(2, 4)),
                vocab=int(_log(rng, 4000, 50000)))


# ---- inputs ---------------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator("cuda").manual_seed(seed)


def _tokens(case, g, batch):
    """Packed documents: uniform tokens, an end-of-document id about every 1024."""
    ids = torch.randint(0, case["vocab"], (batch, case["seq"]), device="cuda", generator=g)
    ends = torch.rand(batch, case["seq"], device="cuda", generator=g) < 1.0 / 1024
    return ids.masked_fill_(ends, case["vocab"] - 1)


def _drop(labels, share, g):
    if share > 0:
        labels = labels.masked_fill(torch.rand(labels.shape, device="cuda", generator=g) < share, IGNORE)
    return labels


def _model(case, seed):
    cfg = dict(num_layers=case["layers"], num_heads=case["heads"], num_kv_heads=case["kv_heads"], emb_dim=case["emb"],
               head_dim=128, vocab_size=case["vocab"], ffn_dim=case["ffn"])
    torch.manual_seed(seed)
    with torch.device("cuda"):
        model = build_model("qwen3_dense" if case["qk_norm"] else "llama3_2", cfg)
        model.init_weights()
    return model


def _prepare_step(case, seed):
    g = _gen(seed + 1)
    model = _model(case, seed)
    batches = []
    for _ in range(case["micro"]):
        ids = _tokens(case, g, case["batch"])
        batches.append({"input_ids": ids, "labels": ids.clone()})
    opt = build_optimizer(model, "adamw", ADAMW)
    ddp = DDP(model, OneRank(), "dp", bucket_mb=25) if case["ddp"] else None
    for p, shadow in model.engine().shadow_pairs():
        opt.attach_shadow(p, shadow)
    obj = build_objective("AR", {"ignore_index": IGNORE, "fused_linear_ce": True, "ce_chunk_size": case["chunk"]})
    return Program(kind="step", model=model, opt=opt, ddp=ddp, obj=obj, batches=batches, params=list(model.parameters()))


def _run_step(s):
    model, opt, ddp, obj, batches = s["model"], s["opt"], s["ddp"], s["obj"], s["batches"]
    scale = 1.0 / len(batches)
    loss = torch.zeros((), device="cuda")
    for i, batch in enumerate(batches):
        if ddp is not None:
            ddp.requires_sync = i == len(batches) - 1
        with torch.autocast(device_type="cuda", dtype=torch.bfloat16):
            part = obj.compute_loss(model, batch, loss_scale=scale)
        part.backward()
        loss += part.detach()
    if ddp is not None:
        ddp.sync()
        norm, coef = ddp.norm_and_coef(1.0)
        opt.set_grad_scale(coef)
        opt.step()
        opt.zero_grad()
        return loss, norm, ddp.reducer.flat, model.token_emb.weight
    norm = clip_grad_norm(s["params"], OneRank(), 1.0)
    opt.step()
    grads = [p.grad for p in s["params"]]
    opt.zero_grad()
    return [loss, norm, model.token_emb.weight, *grads]


def _prepare_forward(case, seed):
    g = _gen(seed + 1)
    model = _model(case, seed)
    model.engine()
    ids = _tokens(case, g, case["batch"])
    labels = _drop(ids.clone(), case.get("ignored", 0.0), g)
    return dict(kind=case["kind"], model=model, ids=ids, labels=labels, chunk=case.get("chunk"))


@torch.no_grad()
def _run_eval(s):
    model = s["model"]
    with torch.autocast(device_type="cuda", dtype=torch.bfloat16):
        hidden = model(s["ids"], return_final_hidden=True)
        loss = fused_linear_cross_entropy(hidden, model.lm_head.weight, shift_labels(s["labels"], IGNORE), IGNORE, s["chunk"])
    return loss, hidden


@torch.no_grad()
def _run_logits(s):
    return s["model"](s["ids"])


def _prepare_linear_ce(case, seed):
    g = _gen(seed)
    h = torch.randn(case["rows"], case["dim"], device="cuda", generator=g).bfloat16().requires_grad_()
    w = torch.randn(case["vocab"], case["dim"], device="cuda", generator=g) * 0.02
    if case["weight"] == "bf16":
        w = w.bfloat16()
    y = torch.randint(0, case["vocab"], (case["rows"],), device="cuda", generator=g)
    return dict(kind="linear_ce", h=h, w=w.requires_grad_(), y=_drop(y, case["ignored"], g), chunk=case["chunk"])


def _run_linear_ce(s):
    s["h"].grad = s["w"].grad = None
    loss = fused_linear_cross_entropy(s["h"], s["w"], s["y"], IGNORE, s["chunk"])
    loss.backward()
    return loss.detach(), s["h"].grad, s["w"].grad


def _prepare_attention(case, seed):
    g = _gen(seed)

    def normal(seq, heads):
        return torch.randn(case["batch"], seq, heads, 128, device="cuda", generator=g).bfloat16()

    q = normal(case["seq"], case["heads"]).requires_grad_()
    k, v = (normal(case["kv_seq"], case["kv_heads"]).requires_grad_() for _ in range(2))
    return dict(kind="attention", q=q, k=k, v=v, g=normal(case["seq"], case["heads"]), causal=case["causal"])


def _run_attention(s):
    q, k, v = s["q"], s["k"], s["v"]
    q.grad = k.grad = v.grad = None
    out = flash_attention(q, k, v, causal=s["causal"])
    out.backward(s["g"])
    return out.detach(), q.grad, k.grad, v.grad


def _shapes(case):
    D, nq, nkv, F = case["emb"], case["heads"] * 128, case["kv_heads"] * 128, case["ffn"]
    block = [(D,), (nq, D), (nkv, D), (nkv, D), (128,), (128,), (D, nq), (D,), (F, D), (F, D), (D, F)]
    return [(case["vocab"], D)] + block * case["blocks"] + [(D,)]


def _prepare_optimizer(case, seed):
    g = _gen(seed)
    params = []
    for shape in _shapes(case):
        p = torch.nn.Parameter(torch.randn(shape, device="cuda", generator=g) * 0.02 if len(shape) > 1
                               else torch.ones(shape, device="cuda"))
        p.grad = torch.randn(shape, device="cuda", generator=g) * 1e-3
        params.append(p)
    return dict(kind="optimizer", params=params, opt=build_optimizer(None, "adamw", ADAMW, params=params))


def _run_optimizer(s):
    norm = clip_grad_norm(s["params"], OneRank(), 1.0)
    s["opt"].step()
    return [norm, *(p.detach() for p in s["params"])]


_PREPARE = {"step": _prepare_step, "eval": _prepare_forward, "logits": _prepare_forward, "linear_ce": _prepare_linear_ce,
            "attention": _prepare_attention, "optimizer": _prepare_optimizer}
_RUN = {"step": _run_step, "eval": _run_eval, "logits": _run_logits, "linear_ce": _run_linear_ce,
        "attention": _run_attention, "optimizer": _run_optimizer}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state["kind"]](state)


# ---- what a pass cannot do without ----------------------------------------------------------------------------------
def _sizes(case):
    """(weights of the block matrices and the head, all parameters)"""
    D, nq, nkv = case["emb"], case["heads"] * 128, case["kv_heads"] * 128
    block = D * (nq + 2 * nkv) + nq * D + 3 * D * case["ffn"]
    matmul = case["layers"] * block + case["vocab"] * D
    return matmul, matmul + case["layers"] * (2 * D + (256 if case["qk_norm"] else 0)) + D


def work(case):
    kind = case["kind"]
    if kind in ("step", "eval", "logits"):
        matmul, params = _sizes(case)
        tokens = case["batch"] * case["seq"] * case.get("micro", 1)
        causal = 2 * case["seq"] * case["heads"] * 128 * case["layers"]      # Q K^T and P V over the visible half, per token
        if kind == "step":
            # master weights and both moments read and written, gradients written; forward + two products per weight
            return {"bytes": 28 * params + 16 * tokens, "flops": tokens * 3 * (2 * matmul + causal)}
        out = 2 * tokens * (case["vocab"] if kind == "logits" else case["emb"])
        return {"bytes": 2 * params + 12 * tokens * case["emb"] + out, "flops": tokens * (2 * matmul + causal)}
    if kind == "linear_ce":
        n, d, v = case["rows"], case["dim"], case["vocab"]
        w = 2 if case["weight"] == "bf16" else 4
        return {"bytes": 4 * n * d + 2 * w * v * d + 8 * n, "flops": 6 * n * d * v}
    if kind == "attention":
        pairs = case["batch"] * case["heads"] * case["seq"] * case["kv_seq"] * (0.5 if case["causal"] else 1)
        rows_q = case["batch"] * case["seq"] * case["heads"] * 128
        rows_k = case["batch"] * case["kv_seq"] * case["kv_heads"] * 128
        return {"bytes": 2 * (4 * rows_q + 4 * rows_k), "flops": 12 * 128 * pairs}
    n = sum(math.prod(s) for s in _shapes(case))
    return {"bytes": 32 * n, "flops": 15 * n}


def tolerance(case):
    """Measured against the same pass in fp32 (PyTorch ops, TF32 off) and, for the optimizer, in fp64.  A training step's
    gradients are 1.1 to 1.5 % off (activations, scores and dlogits are rounded to bf16 layer after layer), the updated table
    0.1 %, the loss 5e-5; single elements of the small gradients next to a large one by about the flat buffer's own rms.
    Hidden states and logits: 1.1 %, elements 0.06.  Loss head: 0.35 %, elements 0.01.  Attention: 0.25 %, elements 0.08.
    Optimizer: norm 5e-7, weights 4e-8."""
    kind = case["kind"]
    if kind == "step":
        return {"rel": 0.03, "max": 0.99}
    if kind in ("eval", "logits"):
        return {"rel": 0.03, "max": 0.25}
    if kind == "linear_ce":
        return {"rel": 0.012, "max": 0.05}
    if kind == "attention":
        return {"rel": 0.01, "max": 0.3}
    return {"rel": 2e-6, "max": 1e-5}
