"""Prompts through the engine whose attention takes the tcgen05 kernels: that it does, and what it gives against the kernels it
replaces.  The latent attention's forms have the same bits; the windowed attention's sum in another order (a layer's difference is a
few bfloat16 roundings, 2^-8 each, of activations that two more layers pass on: 2 % of the logits' norm)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _logits(config, lens, seed=3):
    import transformer_b200 as tb
    from transformer_b200.csrc import lib
    engine = tb.random_model(config, seed=seed, dtype="bfloat16", std=0.05, max_tokens=sum(lens) + 64 * len(lens), max_slots=len(lens))
    g = torch.Generator().manual_seed(seed)
    prompts = [torch.randint(0, config["vocab"], (n,), generator=g).tolist() for n in lens]
    with lib.timing() as t:
        out = engine.step([engine.open() for _ in lens], prompts, want=[list(range(n)) for n in lens]).float().clone()
    assert not lib.gemm_tc_status()
    return out, t.calls


def _salepel(heads, rank, rot):
    att = {"heads": heads, "dim": 32, "rot_dim": rot, "vdim": 32, "kv_rank": rank, "q_rank": 64, "mask": {"size": 200},
           "rot": {"base": 10000.0, "dims": rot}, "scale": (32 + rot) ** -0.5}
    mlp = {"kind": "moe", "router": {"experts": 4, "identity": 1, "top": 2}, "expert": {"ff": 64, "limit": 7.0}}
    return {"architecture": "Salepel", "vocab": 320, "width": 128, "norm": {"eps": 1e-6}, "embedding": {"scale": 1.0}, "max_context": 1024,
            "layers": [{"type": "latent_attention", "mixer": att, "mlp": mlp}] * 2}


@pytest.mark.parametrize("heads,rank,rot", [(8, 256, 32), (16, 512, 64), (6, 256, 64)])
def test_latent_prompts(monkeypatch, heads, rank, rot):
    from transformer_b200.parts import latent_attention
    config, lens = _salepel(heads, rank, rot), [530, 301, 77]
    got, calls = _logits(config, lens)
    assert calls.get("tb_latent_attention_tc_bf16")
    monkeypatch.setattr(latent_attention, "tc_pays", lambda ctx, m: False)
    want, calls = _logits(config, lens)
    assert "tb_latent_attention_tc_bf16" not in calls
    assert bool(torch.isfinite(got).all()) and torch.equal(got, want)


@pytest.mark.parametrize("heads,kv_heads,window,cap", [(8, 2, 300, 30.0), (4, 4, 4096, 0.0)])
def test_windowed_prompts(monkeypatch, heads, kv_heads, window, cap):
    from transformer_b200.parts import attention
    att = {"heads": heads, "kv_heads": kv_heads, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": window, "keep_first": 4},
           "rot": {"base": 10000.0, "dims": 64}}
    if cap:
        att["softcap"] = cap
    config = {"architecture": "Zufadra", "vocab": 320, "width": 256, "norm": {"eps": 1e-6}, "residual_mult": 0.5, "logit_scale": 0.5,
              "embedding": {"scale": 8.0, "bigram": {"buckets": 1021, "mul_prev": 31, "mul_cur": 7}}, "max_context": 1024,
              "layers": [{"type": "attention", "mixer": att, "mlp": {"kind": "dense", "ff": 512}}] * 2}
    lens = [700, 401]
    got, calls = _logits(config, lens)
    assert calls.get("tb_attention_tc_window_bf16")
    monkeypatch.setattr(attention, "window_tcgen05_pays", lambda ctx, m, window: False)
    want, calls = _logits(config, lens)
    assert "tb_attention_tc_window_bf16" not in calls
    assert float((got - want).norm()) <= 0.02 * float(want.norm())
