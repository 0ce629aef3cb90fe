"""Collective helpers, packed weight broadcast, vocab-parallel top-k, routed-expert traces."""

import os
import sys

import pytest
import torch
import torch.distributed as dist

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__))))
from test_parallel_cpu import _spawn  # noqa: E402


def test_pack_and_unpack_buckets():
    from rl_b200.distributed.collectives import pack_tensors, unpack_bucket

    ts = [("a", torch.arange(10, dtype=torch.float32)), ("b", torch.ones(3, 5, dtype=torch.bfloat16)), ("c", torch.arange(7, dtype=torch.int64)),
          ("big", torch.randn(1000))]
    got = {}
    buckets = list(pack_tensors(ts, bucket_bytes=128))
    assert len(buckets) >= 3
    for manifest, buf in buckets:
        assert all(off % 16 == 0 for _, _, _, off, _ in manifest)
        for n, t in unpack_bucket(manifest, buf):
            got[n] = t.clone()
    for n, t in ts:
        assert torch.equal(got[n], t) and got[n].dtype == t.dtype


def _coll_worker(rank, world):
    from rl_b200.distributed.collectives import gather_jagged_object_lists, packed_broadcast, rebalance_nd_tensor
    from rl_b200.parallel.tensor import TP
    from rl_b200.parallel.vocab import vocab_parallel_argmax, vocab_parallel_topk

    t = torch.full((rank + 1, 3), float(rank))
    full = rebalance_nd_tensor(t)
    objs = gather_jagged_object_lists([f"r{rank}-{i}" for i in range(rank + 1)])
    torch.manual_seed(0)
    src = [("w", torch.randn(64, 8)), ("b", torch.arange(5))] if rank == 0 else None
    recv = {n: x.clone() for n, x in packed_broadcast(src, 0, bucket_bytes=1024)}
    z = torch.randn(6, 32, generator=torch.Generator().manual_seed(1))
    tp = TP(None, rank, world)
    v, i = vocab_parallel_topk(z[:, rank * 16 : (rank + 1) * 16], 5, tp, rank * 16)
    rv, ri = torch.topk(z, 5, dim=-1)
    am = vocab_parallel_argmax(z[:, rank * 16 : (rank + 1) * 16], tp, rank * 16)
    return dict(full=full.tolist(), objs=objs, w=float(recv["w"].sum()), b=recv["b"].tolist(),
                topk=bool(torch.equal(i, ri) and torch.allclose(v, rv)), argmax=bool(torch.equal(am, z.argmax(-1))))


def test_collectives_packed_broadcast_and_vocab_topk():
    out = _spawn(_coll_worker, 2)
    torch.manual_seed(0)
    w = torch.randn(64, 8)
    for r in (0, 1):
        assert out[r]["full"] == [[0.0] * 3, [1.0] * 3, [1.0] * 3]
        assert out[r]["objs"] == ["r0-0", "r1-0", "r1-1"]
        assert abs(out[r]["w"] - float(w.sum())) < 1e-5 and out[r]["b"] == [0, 1, 2, 3, 4]
        assert out[r]["topk"] and out[r]["argmax"]


def test_routing_trace_capture_and_replay():
    from rl_b200.models.config import preset
    from rl_b200.models.transformer import PackedBatch, build_model
    from rl_b200.utils import routing_trace as R

    cfg = preset("tiny-llama-oracle", torch_dtype="float32", num_experts=4, num_experts_per_tok=2, moe_intermediate_size=32)
    a, b = build_model(cfg, dtype=torch.float32, seed=1), build_model(cfg, dtype=torch.float32, seed=2)
    batch = PackedBatch.from_padded(torch.randint(0, cfg.vocab_size, (2, 9)), torch.tensor([9, 6]))
    a.hidden_states(batch)
    tr = R.capture(a)
    b.hidden_states(batch)
    assert R.agreement(tr, R.capture(b)) < 0.9     # different routers choose differently
    R.replay(b, tr)
    b.hidden_states(batch)
    assert R.agreement(tr, R.capture(b)) == 1.0
    R.replay(b, None)
    assert b.layers[0].mlp.forced_routing is None


def test_worker_and_generation_satisfy_the_interfaces():
    import torch

    from rl_b200.models.config import ModelConfig
    from rl_b200.policy.interfaces import ColocatablePolicyInterface, GenerationInterface, PolicyInterface, ValueInterface
    from rl_b200.policy.worker import PolicyWorker

    mc = ModelConfig(vocab_size=64, hidden_size=32, intermediate_size=64, num_hidden_layers=1, num_attention_heads=4, num_key_value_heads=2,
                     head_dim=8, torch_dtype="float32")
    w = PolicyWorker(dict(precision="float32", train_global_batch_size=2, train_micro_batch_size=1, max_total_sequence_length=32,
                          optimizer=dict(name="torch.optim.AdamW", kwargs=dict(lr=1e-3)),
                          generation=dict(max_new_tokens=4, kv_cache_tokens=256, block_size=4, max_running=4)), model_cfg=mc, init_reference_model=False)
    assert isinstance(w, PolicyInterface) and isinstance(w, ColocatablePolicyInterface) and isinstance(w, ValueInterface)
    assert isinstance(w.build_generation(), GenerationInterface) and not isinstance(object(), PolicyInterface)


def test_flops_formulas_per_architecture():
    """Component arithmetic checked by hand on small shapes, and the families against each other."""
    from rl_b200.utils import flops as FL

    # one layer, d = 8, 2 heads of 4, 1 kv head, seq 4: projections 2*4*8*(8+8) + 2*4*8*8 = 1536, causal core 2*2*16*8/2 = 256
    assert FL.attention_flops(4, 8, 2, 1, 4) == 1536 + 256
    assert FL.attention_flops(4, 8, 2, 1, 4, causal=False) == 1536 + 512
    assert FL.mlp_flops(4, 8, 16) == 2 * 4 * 8 * 16 * 3 and FL.mlp_flops(4, 8, 16, gated=False) == 2 * 4 * 8 * 16 * 2
    assert FL.moe_flops(4, 8, 16, 2, 8) == 2 * 4 * 8 * 8 + 2 * FL.mlp_flops(4, 8, 16)
    llama = dict(model_type="llama", hidden_size=8, num_hidden_layers=3, num_attention_heads=2, num_key_value_heads=1, head_dim=4,
                 intermediate_size=16, vocab_size=32)
    want = 3 * (FL.attention_flops(4, 8, 2, 1, 4) + FL.mlp_flops(4, 8, 16)) + 2 * 4 * 8 * 32
    assert FL.model_flops(llama, 4, backward=False) == want and FL.model_flops(llama, 4, batch=5) == 15 * want
    moe = dict(llama, model_type="qwen3_moe", num_experts=8, num_experts_per_tok=2, moe_intermediate_size=4)
    assert FL.model_flops(moe, 4, backward=False) == 3 * (FL.attention_flops(4, 8, 2, 1, 4) + FL.moe_flops(4, 8, 4, 2, 8)) + 2 * 4 * 8 * 32
    ds = dict(model_type="deepseek_v3", hidden_size=16, num_hidden_layers=4, num_attention_heads=2, q_lora_rank=8, kv_lora_rank=4,
              qk_nope_head_dim=4, qk_rope_head_dim=2, v_head_dim=4, first_k_dense_replace=1, intermediate_size=32, moe_intermediate_size=8,
              n_routed_experts=8, n_shared_experts=1, num_experts_per_tok=2, vocab_size=64)
    attn = FL.mla_attention_flops(4, 16, 2, 8, 4, 4, 2, 4)
    want = 4 * attn + FL.mlp_flops(4, 16, 32) + 3 * FL.moe_flops(4, 16, 8, 2, 8, 8) + 2 * 4 * 16 * 64
    assert FL.model_flops(ds, 4, backward=False) == want
    hyb = dict(model_type="nemotron_h", hidden_size=16, hybrid_override_pattern="M*-M", num_attention_heads=2, num_key_value_heads=1, head_dim=8,
               mamba_num_heads=4, mamba_head_dim=8, ssm_state_size=8, n_groups=2, conv_kernel=4, intermediate_size=32, vocab_size=64)
    assert FL.model_flops(hyb, 4, backward=False) == (2 * FL.mamba2_flops(4, 16, 32, 8, 2, 4, 4) + FL.attention_flops(4, 16, 2, 1, 8)
                                                       + FL.mlp_flops(4, 16, 32, gated=False) + 2 * 4 * 16 * 64)
    # the packed-batch estimate used for MFU agrees with the per-sequence formula on a dense model
    from rl_b200.models.config import ModelConfig

    mc = ModelConfig(model_type="llama", vocab_size=32, hidden_size=8, intermediate_size=16, num_hidden_layers=3, num_attention_heads=2,
                     num_key_value_heads=1, head_dim=4)
    assert FL.transformer_flops(mc, 4, 4, backward=False) == pytest.approx(FL.model_flops(llama, 4, backward=False))


def test_native_build_sees_included_sources(tmp_path):
    """A source that another one includes (the head-dimension-64 instantiations) is part of what that one was built from."""
    from rl_b200.csrc.build import _digest

    (tmp_path / "a.cu").write_text("int a;\n")
    (tmp_path / "a_d64.cu").write_text('#define RLB_HD 64\n#include "a.cu"\n')
    before = _digest(tmp_path / "a_d64.cu", [])
    (tmp_path / "a.cu").write_text("int b;\n")
    assert _digest(tmp_path / "a_d64.cu", []) != before


def test_gradients_that_begin_anew():
    """After ``begin_grads`` every use sees zeros: a parameter that a backward pass reached, one that none did, and a small one."""
    import torch

    from rl_b200.models.transformer import FlatParams
    from rl_b200.ops import functional as F

    m = torch.nn.Module()
    m.used, m.idle, m.norm = (torch.nn.Parameter(torch.randn(*s)) for s in ((300, 300), (300, 300), (300,)))
    flat = FlatParams(m)
    flat.attach_grad_buffer().fill_(float("nan"))
    flat.begin_grads()
    assert m.used.grad_stale and m.idle.grad_stale and not m.norm.grad_stale and not m.norm.main_grad.any()
    out, add = F.grad_output(m.used, 0)
    assert add and not out.any()
    m.used.grad_stale = True
    out, add = F.grad_output(m.used, 5)
    assert not add and F.grad_output(m.used, 5)[1]
    out.fill_(2.0)
    m.norm.grad = torch.ones(300)
    flat.fold_autograd_grads()
    assert bool((m.used.main_grad == 2).all()) and not m.idle.main_grad.any() and bool((m.norm.main_grad == 1).all())


def test_deferred_metrics_and_packing_without_a_wait():
    """Metrics are made at the first look, additions made before it stay; lengths on the host give the same pack as lengths on the device."""
    import pickle

    import torch

    from rl_b200.algorithms.utils import DeferredMetrics
    from rl_b200.models.transformer import PackedBatch

    made = []
    fresh = lambda: DeferredMetrics(torch.tensor([1.0, 2.0]), lambda v: (made.append(1), dict(a=v[0], b=v[1]))[1])      # noqa: E731
    m = fresh()
    m["lr"] = 3.0
    assert not made
    want = dict(a=1.0, b=2.0, lr=3.0)
    assert m["a"] == 1.0 and dict(m) == want and {**m} == want and sorted(m) == ["a", "b", "lr"] and len(made) == 1
    for look in (lambda x: dict(x), lambda x: {**x}, lambda x: pickle.loads(pickle.dumps(x)), lambda x: dict(x.items()), lambda x: x.copy(), lambda x: {} | x):
        assert look(fresh()) == dict(a=1.0, b=2.0)
    d = dict(z=0)
    d.update(fresh())
    assert d == dict(z=0, a=1.0, b=2.0) and "a" in fresh() and len(fresh()) == 2 and fresh().get("b") == 2.0 and isinstance(fresh(), dict)
    assert not (fresh() != dict(a=1.0, b=2.0)) and fresh().popitem() == ("b", 2.0)
    # only a caller that knows its counts on the host gets them: every other one has a plain dict
    from rl_b200.algorithms.loss.loss_functions import NLLLossFn

    counts = torch.tensor([2.0, 5.0])
    call = lambda toks: NLLLossFn()(-torch.rand(2, 4), dict(token_mask=torch.ones(2, 5), sample_mask=torch.ones(2)), counts[0], toks)[1]      # noqa: E731
    assert type(call(counts[1])) is dict
    known = counts[1]
    known.host = 5.0
    assert type(call(known)) is DeferredMetrics and call(known)["num_unmasked_tokens"] == 8
    ids = torch.arange(40).view(4, 10)
    for lens in ([3, 10, 1, 7], [0, 5, 12, 2], [4, 0, 0, 0]):
        t = torch.tensor(lens)
        a, b = PackedBatch.from_padded(ids, t), PackedBatch.from_padded(ids, t, lens)
        assert torch.equal(a.input_ids, b.input_ids) and torch.equal(a.positions, b.positions) and torch.equal(a.cu_seqlens, b.cu_seqlens)
        assert a.max_seqlen == b.max_seqlen and b.rows is not None and a.positions.dtype == b.positions.dtype and a.cu_seqlens.dtype == b.cu_seqlens.dtype
        x = torch.randn(a.input_ids.numel(), 2)
        assert torch.equal(a.unpack(x, 10), b.unpack(x, 10))
        pa, pb = a.pad_to_multiple(8), b.pad_to_multiple(8)
        y = torch.randn(pa.input_ids.numel())
        assert torch.equal(pa.unpack(y, 10), pb.unpack(y, 10))


def test_kept_logits_leave_room(monkeypatch):
    """Logits are kept for a backward pass only where four times their size is free: of this process's share, and, where its allocator would have to
    grow, of what other processes leave."""
    import types

    import torch

    from rl_b200.ops import functional as F

    M, N = 64, 1024
    size, total = 4 * M * N, 100 << 20
    asked = []

    def kept(used, held, free, fraction=1.0, capturing=False, words=N):
        asked.clear()
        now = dict(allocated_bytes=dict(all=dict(current=used)), reserved_bytes=dict(all=dict(current=held)))
        monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: capturing)
        monkeypatch.setattr(torch.cuda, "get_device_properties", lambda d: types.SimpleNamespace(total_memory=total))
        monkeypatch.setattr(torch.cuda.memory, "memory_stats_as_nested_dict", lambda d: now)
        monkeypatch.setattr(torch.cuda, "get_per_process_memory_fraction", lambda d: fraction)
        monkeypatch.setattr(torch.cuda, "mem_get_info", lambda d: (asked.append(1), (free, total))[1])
        z = F._kept_logits(M, words, torch.device("cpu"))
        assert z is None or (z.shape[0] >= M and z.shape[1] == words and z.dtype == torch.float32)
        return z is not None

    assert kept(0, size, 0) and not asked                                    # the allocator has it: nobody is asked
    assert kept(0, 0, 90 << 20) and asked
    assert not kept(0, 0, 4 * size) and kept(0, 0, 4 * size + total // 20 + 1)      # another process holds the rest
    assert not kept(int(0.95 * total) - 4 * size + 1, total, 0) and kept(int(0.95 * total) - 4 * size - 1, total, 0)
    assert not kept(total // 2, total, 0, fraction=0.5)
    assert not kept(0, size, 0, capturing=True) and not kept(0, size, 0, words=N + 4)
