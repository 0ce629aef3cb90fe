"""The native pass through dense decoder layers against the same layers one by one."""

import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = {      # head dimension 64 and 128, grouped queries, biases, norms of queries and keys; contractions below and above 256
    "llama": dict(hidden_size=512, intermediate_size=1024, num_attention_heads=8, num_key_value_heads=2, head_dim=64),
    "qwen3": dict(hidden_size=256, intermediate_size=320, num_attention_heads=4, num_key_value_heads=4, head_dim=128, qk_norm=True),
    "biased": dict(hidden_size=192, intermediate_size=320, num_attention_heads=4, num_key_value_heads=1, head_dim=128, attention_bias=True),
}


def _model(name):
    from rl_b200.models.config import preset
    from rl_b200.models.transformer import build_model

    torch.manual_seed(1)
    m = build_model(preset("llama3.2-1b", num_hidden_layers=3, vocab_size=512, **SHAPES[name]), device="cuda", dtype=torch.bfloat16)
    for p in m.parameters():
        p.data.normal_(0.0, 0.05)
        if p.dim() < 2:
            p.data.add_(1.0)
    return m


def _batch(T):
    cut = sorted({0, T // 3, T // 3 + min(1, T), T})
    cu = torch.tensor(cut, dtype=torch.int32, device="cuda")
    pos = torch.cat([torch.arange(b - a, dtype=torch.int32, device="cuda") for a, b in zip(cut, cut[1:])])
    return cu, pos, max(b - a for a, b in zip(cut, cut[1:]))


@pytest.mark.parametrize("name", list(SHAPES))
@pytest.mark.parametrize("T", [1, 40, 256, 257, 700])
@pytest.mark.parametrize("cached", [False, True])
@torch.no_grad()
def test_dense_forward(native_lib, name, T, cached):
    """The same kernels: equal bit for bit, the caches too."""
    from rl_b200.ops import engine_ops as E
    from rl_b200.ops import functional as F
    from rl_b200.ops.dense_forward import dense_forward

    m = _model(name)
    c = m.cfg
    cu, pos, longest = _batch(T)
    h = torch.randn(T, c.hidden_size, generator=torch.Generator("cuda").manual_seed(T), device="cuda").bfloat16()
    at = m.layers[0].self_attn
    caches = [[torch.zeros(T // 16 + 2, at.hkv, 16, c.head_dim, dtype=torch.bfloat16, device="cuda") for _ in range(6)] for _ in range(2)]
    slots = torch.randperm(T, device="cuda")
    first = h.clone()
    kw = dict(slots=slots, k_caches=caches[0][:3], v_caches=caches[0][3:]) if cached else {}
    got = dense_forward(m.layers, h, pos, [m.inv_freq] * 3, cu, longest, **kw)
    assert torch.equal(h, first)
    ref = h
    for i, layer in enumerate(m.layers):
        x = F.rmsnorm(ref, layer.input_layernorm, c.rms_norm_eps)
        qkv = layer.self_attn.project_qkv(x, pos, m.inv_freq, apply_rope=False)
        if cached:
            qkv = E.rope_kv_cache_write(qkv, pos, m.inv_freq, slots, caches[1][i], caches[1][3 + i], at.hq, at.hkv, c.head_dim)
        else:
            qkv = F.rope(qkv, pos, m.inv_freq, at.hq + at.hkv, c.head_dim)
        ref = layer.tail(ref, F.attention_varlen(qkv, cu, longest, at.hq, at.hkv, c.head_dim))
    assert torch.equal(got, ref)
    for a, b in zip(*caches):
        assert torch.equal(a, b)


@torch.no_grad()
def test_dense_forward_leaves_other_layers_alone(native_lib):
    """Hooks, replaced methods, adapters, other types and passes with gradients go layer by layer."""
    from rl_b200.ops.dense_forward import dense_forward

    m = _model("llama")
    cu, pos, longest = _batch(40)
    h = torch.randn(40, 512, device="cuda").bfloat16()
    run = lambda x=h: dense_forward(m.layers, x, pos, [m.inv_freq] * 3, cu, longest)      # noqa: E731
    assert run() is not None
    handle = m.layers[1].mlp.register_forward_hook(lambda *a: None)
    assert run() is None
    handle.remove()
    m.layers[2].self_attn.qkv_lora = object()
    assert run() is None
    m.layers[2].self_attn.qkv_lora = None
    m.layers[0].forward = m.layers[0].forward
    assert run() is None
    del m.layers[0].__dict__["forward"]
    assert run(h.float()) is None and run(h[:, ::2]) is None and run(h[:0]) is None
    with torch.enable_grad():
        assert run() is None
    assert run() is not None
