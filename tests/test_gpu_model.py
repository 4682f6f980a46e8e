"""GPU end-to-end: model loss / gradients on the CUDA kernels (bf16) against the CPU restatement (fp32 math on the
same bf16-rounded weights), for every layer family; an optimizer step; the driver's smoke entry point."""

import pytest
import torch

pytestmark = pytest.mark.gpu

from olmax_b200.activation_checkpointing import NothingSaveable, SaveAnythingExceptTheseNames
from olmax_b200.models import (
    DefaultTransformerConfig,
    DefaultTransformerLayerConfig,
    GemmaTransformerLayerConfig,
    ReorderedNormTransformerLayerConfig,
)
from olmax_b200.nn import LMHeadConfig, MultiheadSelfAttentionConfig, RMSNormConfig, RotaryPositionalEmbeddingConfig
from olmax_b200.optim import AdamWConfig, ConstantSchedule
from olmax_b200.parallel import MeshResource


def _make(dev, layer_cls, qk=False, headwise=True, kv=None, softcap=None, fsoft=None, tie=False, window=None, ac=None):
    attn = MultiheadSelfAttentionConfig(n_heads=4, n_kv_heads=kv, head_dim=128,
                                        rope=RotaryPositionalEmbeddingConfig(theta=10000.0),
                                        qk_norm=RMSNormConfig() if qk else None, use_head_qk_norm=headwise,
                                        logit_softcap=softcap)
    cfg = DefaultTransformerConfig(vocab_size=2048, d_model=512, hidden_size=1024, num_layers=2,
                                   layer=layer_cls(attention=attn), lm_head=LMHeadConfig(logit_softcap=fsoft),
                                   tie_embeddings=tie, scale_embeddings=tie, sliding_window=window,
                                   sliding_window_pattern=2, layer_ac_policy=ac, ce_chunk_rows=256)
    return cfg.build(seed=1, mesh_resource=MeshResource.FSDP(1), device=torch.device(dev))


CASES = {
    "llama": dict(layer_cls=DefaultTransformerLayerConfig),
    "olmo2_full_qk": dict(layer_cls=ReorderedNormTransformerLayerConfig, qk=True, headwise=False),
    "olmo2_head_qk_gqa": dict(layer_cls=ReorderedNormTransformerLayerConfig, qk=True, headwise=True, kv=2),
    "gemma": dict(layer_cls=GemmaTransformerLayerConfig, kv=2, softcap=50.0, fsoft=30.0, tie=True, window=100),
    "llama_remat": dict(layer_cls=DefaultTransformerLayerConfig, ac=NothingSaveable()),
    "gemma_mlp_remat": dict(layer_cls=GemmaTransformerLayerConfig, kv=2, softcap=50.0,
                            ac=SaveAnythingExceptTheseNames(names=["layers.*.mlp"])),
    "olmo2_attention_remat": dict(layer_cls=ReorderedNormTransformerLayerConfig, qk=True, headwise=True,
                                  ac=SaveAnythingExceptTheseNames(names=["layers.*.attention"])),
}


@pytest.mark.parametrize("name", list(CASES))
def test_model_matches_cpu_restatement(name):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from olmax_b200.ops import _lib

    kw = CASES[name]
    torch.manual_seed(0)
    ids = torch.randint(0, 2048, (2, 256))
    labels = torch.roll(ids, -1, 1)
    labels[:, -1] = -100
    mc, mg = _make("cpu", **kw), _make("cuda", **kw)
    mg.store.master.copy_(mc.store.master.to("cuda"))
    mg.store.sync_shadow()
    mc.store.master.copy_(mg.store.shadow.float().cpu())
    mc.store.sync_shadow()
    out = {}
    for m, dev in ((mc, "cpu"), (mg, "cuda")):
        m.store.set_grad_scale(1.0)
        cache = m.get_buffer_cache(256, torch.device(dev))
        loss, _ = m(ids.to(dev), labels.to(dev), cache)
        loss.backward()
        m.store.finish_backward()
        out[dev] = (loss.item(), m.store.grad.float().cpu().clone())
    _lib.check_status()
    assert abs(out["cpu"][0] - out["cuda"][0]) < 5e-3 * abs(out["cpu"][0])
    gc_, gg = out["cpu"][1], out["cuda"][1]
    assert ((gc_ - gg).norm() / gc_.norm()).item() < 4e-2
    for n, h in mc.store.named_parameters():
        a = gc_[h.meta.offset : h.meta.offset + h.meta.numel_local]
        b = gg[h.meta.offset : h.meta.offset + h.meta.numel_local]
        assert ((a - b).norm() / (a.norm() + 1e-20)).item() < 8e-2, n


@pytest.mark.parametrize("used", ["all", "last"])   # outputs that carry a gradient
@pytest.mark.parametrize("widths,bias,joined", [
    ((128, 128), False, True),
    ((384, 128, 256), False, True),
    ((136, 128), False, False),       # rows that are no whole tiles
    ((128, 136, 128), False, False),
    ((128, 128), True, False),        # the biases lie between the weights
])
def test_linears_of_one_input_joined_and_apart(widths, bias, joined, used):
    """``linear_group`` over handles of a parameter store: outputs, dx and the whole flat gradient buffer (the weight that
    follows the group too, which has none) as from calls one by one."""
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from olmax_b200.nn.linear import Linear, linear_group
    from olmax_b200.nn.module import Module, build_module, current_build_context
    from olmax_b200.ops import _lib, functional as F
    from olmax_b200.testing import rel_err

    class Group(Module):
        def __init__(self):
            super().__init__()
            self.mods = torch.nn.ModuleList()
            for i, n in enumerate((*widths, 128)):
                with current_build_context().scope(f"p{i}"):
                    self.mods.append(Linear(256, n, bias=bias))

    group = build_module(Group, seed=3, mesh_resource=MeshResource.FSDP(1), device=torch.device("cuda"))
    mods = list(group.mods)[: len(widths)]
    assert F._joined([m.weight for m in mods]) == joined
    torch.manual_seed(7)
    x0 = torch.randn(2, 100, 256, device="cuda", dtype=torch.bfloat16)
    dys = [torch.randn(2, 100, n, device="cuda", dtype=torch.bfloat16) for n in widths]
    results = []
    for run in (lambda x: linear_group(mods, x), lambda x: tuple(m(x) for m in mods)):
        group.store.set_grad_scale(0.5)
        group.store.grad.zero_()
        x = x0.clone().requires_grad_(True)
        ys = run(x)
        first = 0 if used == "all" else len(widths) - 1
        torch.autograd.backward(ys[first:], dys[first:])
        group.store.finish_backward()
        results.append((ys, x.grad, group.store.grad.clone()))
    (ys, dx, grad), (ys1, dx1, grad1) = results
    for y, y1 in zip(ys, ys1):
        assert rel_err(y, y1.float()) < 4e-3   # one bf16 rounding each, 2^-9 at most
    assert rel_err(dx, dx1.float()) < 1e-2     # apart: one bf16 tensor per weight and their bf16 sums
    assert rel_err(grad, grad1) < 1e-5         # fp32 sums
    tail = group.mods[-1].weight.meta
    assert not grad[tail.offset : tail.offset + tail.numel_local].any()
    _lib.check_status()


def test_gated_mlp_joined_and_apart(monkeypatch):
    """The gated MLP's backward with gate and up as one matrix against the separate GEMMs: dx and every gradient."""
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from olmax_b200.nn.mlp import GatedMLP
    from olmax_b200.nn.module import build_module
    from olmax_b200.ops import _lib, functional as F
    from olmax_b200.testing import rel_err

    mlp = build_module(lambda: GatedMLP(256, 384), seed=3, mesh_resource=MeshResource.FSDP(1), device=torch.device("cuda"))
    assert F._joined((mlp.gate_proj.weight, mlp.up_proj.weight))
    torch.manual_seed(8)
    x0, dy = (torch.randn(200, 256, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    results = []
    for joined in (True, False):
        if not joined:
            monkeypatch.setattr(F, "_joined", lambda handles: False)
        mlp.store.set_grad_scale(1.0)
        mlp.store.grad.zero_()
        x = x0.clone().requires_grad_(True)
        mlp(x).backward(dy)
        mlp.store.finish_backward()
        results.append((x.grad, mlp.store.grad.clone()))
    (dx, grad), (dx1, grad1) = results
    assert rel_err(dx, dx1.float()) < 1e-2 and rel_err(grad, grad1) < 1e-5
    _lib.check_status()


def test_optimizer_step_matches_cpu():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    mc, mg = _make("cpu", DefaultTransformerLayerConfig), _make("cuda", DefaultTransformerLayerConfig)
    mg.store.master.copy_(mc.store.master.to("cuda"))
    mg.store.sync_shadow()
    oc = AdamWConfig(lr=ConstantSchedule(1e-3), weight_decay=0.1, max_grad_norm=1.0, no_decay_modules=["embedding.weight"])
    opt_c, opt_g = oc.build(mc), oc.build(mg)
    g = torch.randn(mc.store.numel_local) * 0.01
    for _ in range(3):
        mc.store.grad.copy_(g)
        mg.store.grad.copy_(g.cuda())
        opt_c.step()
        opt_g.step()
    err = ((mc.store.master - mg.store.master.cpu()).norm() / mc.store.master.norm()).item()
    assert err < 1e-5
    assert abs(opt_c.grad_norm.item() - opt_g.grad_norm.item()) < 1e-3 * opt_c.grad_norm.item()
    assert mg.store.grad.abs().max().item() == 0.0
    assert ((mg.store.shadow.float() - mg.store.master).abs().max() / mg.store.master.abs().max()).item() < 1e-2


def test_smoke_entry_point():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    import __graft_entry__

    __graft_entry__.smoke()
