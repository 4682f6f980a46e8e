"""
Performance cases of the framework on one GPU: what a user has it do, through the calls a user makes.

Three kinds of work, over the sizes of this repository's recipes, tests and benchmark:

* ``train``: one optimizer step through ``Trainer.train_batch``: pinned host ids / labels in, forward, backward, AdamW; back
  come the loss, the updated master weights and the first moments (which carry the step's gradients; those of the
  input embedding are mostly zero rows and are seen through its updated weights).  The wide models are cut in depth
  (``layers``), not in width, so that the state fits several times over.
* ``logits`` / ``loss``: a forward pass without gradients (scoring a prompt, an evaluation batch).
* ``attention``: forward and backward of the attention op on its own, as a custom model built from the ops calls it.

A case is a dict of plain values; :func:`prepare` makes what a program has in hand before the call, :func:`run` makes one
pass, :func:`work` counts what the pass cannot do without.
"""

from __future__ import annotations

import dataclasses
import gc
import math
import tempfile
from pathlib import Path

import torch

from olmax_b200.models import (DefaultTransformerConfig, ReorderedNormTransformerLayerConfig, TransformerRecipeType)
from olmax_b200.nn import MultiheadSelfAttentionConfig, RMSNormConfig
from olmax_b200.ops import functional as F
from olmax_b200.optim import AdamWConfig, ConstantSchedule
from olmax_b200.parallel import MeshResource
from olmax_b200.train import Trainer

HEAD_DIM = 128


def listed():
    return [
        # The two-layer OLMo2-style model of the smoke test: unit-test sized steps, where launches and host time count.
        dict(name="step-smoke", kind="train", recipe="smoke", layers=2, batch=2, seq=512, micro=1, clip=False),
        # A short fine-tuning step of the whole 271M model on 1000 tokens (not a multiple of any tile), with clipping.
        dict(name="step-271M-short", kind="train", recipe="llama_like_271M", layers=16, batch=1, seq=1000, micro=1, clip=True),
        # The 271M recipe's own pre-training micro-batch (64 x 1024 tokens).
        dict(name="step-271M-full", kind="train", recipe="llama_like_271M", layers=16, batch=64, seq=1024, micro=1, clip=True),
        # The headline benchmark's step (OLMo2 7B, 2 x 4096 tokens per micro-batch, two micro-batches), four layers deep.
        dict(name="step-olmo2-7B", kind="train", recipe="olmo2_7B_bench", layers=4, batch=2, seq=4096, micro=2, clip=False),
        # Gemma2-like 27B width: GeGLU, grouped heads, soft-caps, windowed and global attention, tied 256000-row head.
        dict(name="step-gemma2-27B", kind="train", recipe="gemma2_like_27B_bench", layers=2, batch=1, seq=4096, micro=1, clip=True),
        # OLMo2 32B width: 40/8 heads, per-head q/k norm, whole layers recomputed; a ragged sequence length.
        dict(name="step-olmo2-32B", kind="train", recipe="olmo2_32B_bench", layers=2, batch=2, seq=2780, micro=1, clip=False),
        # Scoring one prompt with the 271M model: the logits of 328 tokens.
        dict(name="logits-271M", kind="logits", recipe="llama_like_271M", layers=16, batch=1, seq=328),
        # An evaluation batch of the Llama3 8B width at its full sequence length.
        dict(name="loss-llama3-8B", kind="loss", recipe="llama3_8B", layers=4, batch=1, seq=8192),
        # Attention alone: the smallest calls, the 7B shape, a ragged grouped one, a windowed and soft-capped one.
        dict(name="attn-small", kind="attention", batch=1, seq=384, heads=8, kv_heads=8, window=-1, softcap=0.0),
        dict(name="attn-7B", kind="attention", batch=2, seq=4096, heads=32, kv_heads=32, window=-1, softcap=0.0),
        dict(name="attn-gqa-ragged", kind="attention", batch=3, seq=1515, heads=40, kv_heads=8, window=-1, softcap=0.0),
        dict(name="attn-window-cap", kind="attention", batch=1, seq=8192, heads=32, kv_heads=16, window=4096, softcap=50.0),
    ]


# recipe -> the depths a drawn case may have (bounded by memory: three states fit the card)
_DEPTHS = {"smoke": (1, 6), "llama_like_271M": (4, 16), "llama_like_7B_bench": (1, 4), "olmo2_7B_bench": (1, 4),
           "llama3_8B": (1, 4), "olmo2_32B_bench": (1, 2), "gemma2_like_27B_bench": (1, 2)}


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(["train", "train", "train", "logits", "loss", "attention", "attention"])
        if kind == "attention":
            heads, kv = rng.choice([(4, 4), (8, 8), (16, 4), (32, 32), (32, 8), (32, 16), (40, 8), (64, 8)])
            case = dict(kind=kind, batch=rng.randint(1, 4), seq=_log_int(rng, 128, 8192), heads=heads, kv_heads=kv,
                        window=rng.choice([-1, -1, -1, 128, 1024, 4096]), softcap=rng.choice([0.0, 0.0, 50.0]))
        else:
            recipe = rng.choice(list(_DEPTHS))
            batch = rng.randint(1, 8)
            # the GEMMs take token counts that are multiples of 8
            seq = max(1, _log_int(rng, 128, 8192) * math.gcd(batch, 8) // 8) * 8 // math.gcd(batch, 8)
            case = dict(kind=kind, recipe=recipe, layers=rng.randint(*_DEPTHS[recipe]), batch=batch, seq=seq)
            if kind == "train":
                case.update(micro=rng.randint(1, 2), clip=rng.random() < 0.5)
            if kind == "logits" and batch * seq > 8192:   # fp32 logits are returned whole
                continue
            if batch * seq > 65536 or (kind == "train" and batch * seq < 1000):
                continue
        if _cost(case) <= most:
            return case


# ------------------------------------------------------------------------------------------------------------- models
def _model_config(case):
    if case["recipe"] == "smoke":
        attn = MultiheadSelfAttentionConfig(n_heads=4, head_dim=HEAD_DIM, qk_norm=RMSNormConfig(), use_head_qk_norm=False)
        cfg = DefaultTransformerConfig(vocab_size=4096, d_model=512, hidden_size=1408,
                                       layer=ReorderedNormTransformerLayerConfig(attention=attn), ce_chunk_rows=512)
    else:
        cfg = TransformerRecipeType(case["recipe"]).build_recipe().model
    return dataclasses.replace(cfg, num_layers=case["layers"])


def _matmul_params(cfg):
    """(parameters that enter a matrix product per token, all parameters up to the norm weights)."""
    att = cfg.layer.attention
    kv = att.n_kv_heads or att.n_heads
    layer = cfg.d_model * HEAD_DIM * (2 * att.n_heads + 2 * kv) + 3 * cfg.d_model * cfg.hidden_size
    head = cfg.vocab_size * cfg.d_model
    return cfg.num_layers * layer + head, cfg.num_layers * layer + (1 if cfg.tie_embeddings else 2) * head


def _visible(seq, window):
    """(query, key) pairs of one causal head, keys no further back than ``window``."""
    w = seq if window is None or window < 0 else min(window + 1, seq)
    return w * (w + 1) // 2 + (seq - w) * w


def _attention_flops(batch, seq, heads, window, passes):
    return passes * 4 * HEAD_DIM * batch * heads * _visible(seq, window)


def work(case):
    if case["kind"] == "attention":
        q = case["batch"] * case["seq"] * case["heads"] * HEAD_DIM * 2
        kv = case["batch"] * case["seq"] * case["kv_heads"] * HEAD_DIM * 2
        return {"bytes": 4 * q + 4 * kv,   # q, o, d_o, dq; k, v, dk, dv
                "flops": _attention_flops(case["batch"], case["seq"], case["heads"], case["window"], 3)}
    cfg = _model_config(case)
    att = cfg.layer.attention
    used, params = _matmul_params(cfg)
    micro = case.get("micro", 1)
    tokens = case["batch"] * case["seq"] * micro
    passes = 3 if case["kind"] == "train" else 1
    flops = passes * 2 * used * tokens
    for i in range(cfg.num_layers):
        flops += _attention_flops(case["batch"] * micro, case["seq"], att.n_heads, cfg.window_size_for_layer(i), passes)
    if case["kind"] == "train":
        nbytes = 24 * params + 16 * tokens          # fp32 weights and both moments, read and written; ids and labels
    else:
        nbytes = 2 * used + 8 * tokens              # bf16 weights once
        if case["kind"] == "logits":
            nbytes += 4 * tokens * cfg.vocab_size
        else:
            nbytes += 8 * tokens
    return {"bytes": nbytes, "flops": flops}


def _cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / 50)


# -------------------------------------------------------------------------------------------------------------- passes
def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev).manual_seed(seed)
    if case["kind"] == "attention":
        def rand(heads):
            return torch.randn(case["batch"], case["seq"], heads, HEAD_DIM, generator=gen, device=dev).to(torch.bfloat16)

        q, k, v, d_o = rand(case["heads"]), rand(case["kv_heads"]), rand(case["kv_heads"]), rand(case["heads"])
        return dict(case=case, inputs=[t.requires_grad_(True) for t in (q, k, v)], d_o=d_o)
    gc.collect()   # an earlier model (its parameter store and handles refer to each other) gives its memory back first
    cfg = _model_config(case)
    model = cfg.build(seed=seed, mesh_resource=MeshResource.FSDP(1), device=dev)
    state = dict(case=case, model=model, cache=model.get_buffer_cache(case["seq"], dev))
    shape = (case["batch"], case["seq"])
    batches = []
    for _ in range(case.get("micro", 1)):
        ids = torch.randint(0, cfg.vocab_size, shape, generator=gen, device=dev)
        labels = torch.roll(ids, -1, 1)
        labels[:, -1] = -100   # the last token has no successor
        batches.append((ids, labels))
    if case["kind"] == "train":
        state["batch"] = [(i.cpu().pin_memory(), l.cpu().pin_memory()) for i, l in batches]
        folder = Path(tempfile.gettempdir()) / "olmax_b200_perf"
        optim = AdamWConfig(lr=ConstantSchedule(1e-4), no_decay_modules=["embedding.weight"],
                            max_grad_norm=1.0 if case["clip"] else None)
        trainer = Trainer(work_dir=folder, save_folder=folder, optim=optim)
        state["trainer"] = trainer.setup(model, case["micro"], state["cache"])
        state["momentum"] = _moments(model, trainer.optimizer.exp_avg)
    else:
        state["ids"], state["labels"] = batches[0]
    return state


def _moments(model, flat):
    """Views of the flat first moments: the matrices and the norm weights of every unit (layer, head) side by side."""
    views = []
    for unit in model.store.units[1:]:
        kinds = []
        for h in unit.params:
            m = h.meta
            if kinds and kinds[-1][0] == len(m.shape):
                kinds[-1][2] = m.offset + m.numel_local
            else:
                kinds.append([len(m.shape), m.offset, m.offset + m.numel_local])
        views += [flat[start:end] for _, start, end in kinds]
    return views


def run(state):
    kind = state["case"]["kind"]
    if kind == "attention":
        c = state["case"]
        q, k, v = state["inputs"]
        o = F.attention(q, k, v, causal=True, window=c["window"], softcap=c["softcap"])
        return (o.detach(), *torch.autograd.grad(o, (q, k, v), state["d_o"]))
    model, cache = state["model"], state["cache"]
    if kind == "train":
        trainer = state["trainer"]
        loss = trainer.train_batch(state["batch"])
        return {"loss": loss, "weights": model.store.master, "momentum": state["momentum"]}
    with torch.no_grad():
        if kind == "logits":
            return model(state["ids"], cache=cache)
        loss, _ = model(state["ids"], state["labels"], cache)
        return loss


def tolerance(case):
    # bf16 tensors between the ops, fp32 sums.  Against the same pass with fp32 tensors between the ops (weights rounded to
    # bf16 alike) the present kernels are off by: attention 0.002-0.0033 (largest difference 0.13), loss 2e-5, logits of 16
    # layers 0.013 (0.073), moments 0.008-0.019 (0.45), updated weights 0.0005.
    if case["kind"] == "attention":
        return {"rel": 1.2e-2, "max": 0.5}
    if case["kind"] == "loss":
        return {"rel": 1e-4, "max": 1e-4}
    if case["kind"] == "logits":
        return {"rel": 3e-2, "max": 0.3}
    return {"rel": 3e-2, "max": 0.99}
