"""The work that is timed when this framework is made faster: generation, prefill, log-probabilities and training steps as the recipes and the
benchmarks of this repository have it do, at random weights of the preset architectures. ``listed`` names them, ``draw`` gives more of the same
ranges, ``prepare`` builds what a program holds before the call, ``run`` is one call through the public entry points, ``exact`` the same numbers
in float64 from plain PyTorch.

Every model's next token is likely the one that follows its last token in a fixed permutation (the output head is the permuted embedding), as a
trained model is sure of most of its tokens; the layers add about as much to the residual stream as the embedding holds.
"""

import math
import random
import zlib

import torch

from rl_b200.algorithms.loss.loss_functions import ClippedPGLossFn, NLLLossFn
from rl_b200.distributed.batched_data_dict import BatchedDataDict
from rl_b200.engine.engine import GenerationEngine, SamplingParams
from rl_b200.models.config import preset
from rl_b200.models.transformer import build_model
from rl_b200.policy.worker import PolicyWorker

LR, DECAY, BETAS, EPS, MAX_NORM = 3e-7, 0.01, (0.9, 0.999), 1e-8, 1.0
SHARE = {"llama3.1-8b": 0.55, "llama3.2-1b": 0.87, "qwen3-30b-a3b": 0.97, "gadarax-1b": 1.0}     # of the final hidden state that points along its token's embedding
BLOCK = 64                 # tokens of a cache page
EXACT_FLOPS = 2.5e14       # most float64 work of ``exact``: some ten seconds


def listed():
    return [
        # one user's short question to the smallest recipe model: launches and latency
        dict(name="chat-1b", kind="generate", model="llama3.2-1b", layers=16, prompts=1, samples=1, length=45, new_tokens=16, temperature=0.0),
        # the headline GRPO rollout: 8 prompts of 256 tokens, 8 samples of each, the first part of the responses
        dict(name="rollout-8b", kind="generate", model="llama3.1-8b", layers=32, prompts=8, samples=8, length=256, new_tokens=24, temperature=1.0),
        # sampling in groups on long prompts: decoding is bound by the cache
        dict(name="rollout-8b-long", kind="generate", model="llama3.1-8b", layers=32, prompts=3, samples=16, length=4001, new_tokens=16, temperature=1.0),
        # evaluation of a mixture-of-experts policy: greedy, every prompt its own; a quarter of the layers
        dict(name="eval-moe", kind="generate", model="qwen3-30b-a3b", layers=12, prompts=32, samples=1, length=300, new_tokens=16, temperature=0.0),
        # serving a layer-list model
        dict(name="serve-layer-list", kind="generate", model="gadarax-1b", layers=12, prompts=16, samples=1, length=700, new_tokens=24, temperature=0.0),
        # ragged prompts of thousands of tokens through the engine's step function
        dict(name="prefill-8b", kind="prefill", model="llama3.1-8b", layers=32, prompts=5, length=3000),
        # the log-probability phase of the headline step, packed into one 20480-token pass
        dict(name="logprobs-8b", kind="logprobs", model="llama3.1-8b", layers=32, sequences=16, length=1200, budget=20480),
        # a small batch of short sequences, as in the smallest recipes' validation
        dict(name="logprobs-1b-short", kind="logprobs", model="llama3.2-1b", layers=16, sequences=4, length=60, budget=0),
        # the training phase of the headline step in 5120-token micro-batches, on four of its layers
        dict(name="train-grpo", kind="train", model="llama3.1-8b", layers=4, sequences=16, length=1000, budget=5120, loss="grpo"),
        # supervised fine-tuning of the smallest recipe model: tied embeddings, heads of 64
        dict(name="train-sft-1b", kind="train", model="llama3.2-1b", layers=16, sequences=8, length=500, budget=4096, loss="sft"),
        # long-context fine-tuning: attention is a large part
        dict(name="train-long", kind="train", model="llama3.1-8b", layers=2, sequences=2, length=7600, budget=8192, loss="sft"),
        # a mixture-of-experts policy, two of its layers, on the experts that the rollout chose
        dict(name="train-moe", kind="train", model="qwen3-30b-a3b", layers=2, sequences=8, length=1000, budget=8192, loss="grpo"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["generate", "generate", "prefill", "logprobs", "train", "train"])
    if kind == "generate":
        model, layers = rng.choice([("llama3.2-1b", 16), ("llama3.1-8b", 32), ("qwen3-30b-a3b", 12), ("gadarax-1b", 12)])
        length = _log(rng, 20, 4000)
        most = max(1, min(64, 24000 // length))          # prompts that are prefilled
        prompts = _log(rng, 1, most)
        samples = 1 if model == "gadarax-1b" else rng.choice([1, 1, 4, max(1, 64 // prompts)])
        samples = max(1, min(samples, 64 // prompts))
        return dict(kind=kind, model=model, layers=layers, prompts=prompts, samples=samples, length=length, new_tokens=rng.randint(2, 20),
                    temperature=1.0 if samples > 1 else 0.0)
    if kind == "prefill":
        model, layers = rng.choice([("llama3.2-1b", 16), ("llama3.1-8b", 32)])
        length = _log(rng, 30, 7000)
        return dict(kind=kind, model=model, layers=layers, prompts=_log(rng, 1, max(1, min(32, 15000 // length))), length=length)
    if kind == "logprobs":
        model, layers = rng.choice([("llama3.2-1b", 16), ("llama3.1-8b", 32)])
        length = _log(rng, 40, 4000)
        return dict(kind=kind, model=model, layers=layers, sequences=_log(rng, 1, max(1, min(64, 18000 // length))), length=length,
                    budget=rng.choice([0, 8192, 20480]))
    model, layers = rng.choice([("llama3.2-1b", 16), ("llama3.1-8b", 2), ("llama3.1-8b", 4), ("qwen3-30b-a3b", 2)])
    length = _log(rng, 40, 7000)
    most = 15000 if layers == 4 else 12000 if layers == 2 else 8000
    return dict(kind=kind, model=model, layers=layers, sequences=_log(rng, 1, max(1, min(32, most // length))), length=length,
                budget=rng.choice([4096, 5120, 8192]), loss=rng.choice(["grpo", "sft"]))


# ---------------------------------------------------------------------------------------------------------------- inputs
def _config(case):
    return preset(case["model"], num_hidden_layers=case["layers"])


def _lengths(case, n):
    """Ragged lengths around the case's, the same for every seed."""
    r = random.Random(case["length"] * 1009 + n)
    return [max(2, int(case["length"] * r.uniform(0.8, 1.2))) for _ in range(n)]


def _successor(cfg):
    """The token that likely follows each token (itself where the output head is the embedding)."""
    if cfg.tie_word_embeddings:
        return torch.arange(cfg.vocab_size, device="cuda")
    return torch.randperm(cfg.vocab_size, device="cuda", generator=torch.Generator("cuda").manual_seed(17))


def _weight(case, cfg, name, shape, seed):
    """The values of one parameter in bf16. The likely token's logit is some 20 where tokens are sampled, so that hardly any is drawn by a hair,
    and 11 elsewhere: a probability of about 0.3."""
    def normal(std, name=name, shape=shape):
        g = torch.Generator("cuda").manual_seed(seed * 1000003 + zlib.crc32(name.encode()))
        return torch.empty(tuple(shape), dtype=torch.bfloat16, device="cuda").normal_(0.0, std, generator=g)

    leaf, peak = name.rsplit(".", 1)[-1], (20.0 if case.get("temperature") else 11.0) / cfg.hidden_size / SHARE[case["model"]]
    stream = 0.0138 if cfg.is_mixer else peak if cfg.tie_word_embeddings else 0.5
    if leaf == "embed_tokens":
        return normal(stream)
    if leaf == "lm_head":
        w = torch.empty(tuple(shape), dtype=torch.bfloat16, device="cuda")
        w[_successor(cfg)] = normal(0.5, "embed_tokens") * (peak / 0.5)
        return w
    if leaf == "alpha":
        return torch.full(tuple(shape), 0.5, dtype=torch.bfloat16, device="cuda")
    if len(shape) < 2:
        return normal(0.02) if leaf.endswith("bias") else normal(0.05) + 1
    if leaf in ("o_proj", "down_proj", "out_proj"):      # the mean of a token's experts is smaller than one wide unit's output
        more = 4.0 if len(shape) == 3 else 1.0
        return normal(0.02 * more / math.sqrt(2 * cfg.num_hidden_layers) * (1.0 if cfg.is_mixer else stream))
    return normal(0.05 if leaf == "router" else 0.02)


@torch.no_grad()
def _fill(model, case, cfg, seed):
    for name, p in model.named_parameters():
        p.data.copy_(_weight(case, cfg, name, p.shape, seed))


def _tokens(cfg, lengths, seed):
    """Token ids [n, longest] on the host and their lengths; seven in ten tokens follow their predecessor as the model expects."""
    g = torch.Generator().manual_seed(seed)
    n, S = len(lengths), max(lengths)
    follow, nxt = torch.rand((n, S), generator=g) < 0.7, _successor(cfg).cpu()
    ids = torch.randint(0, cfg.vocab_size, (n, S), generator=g)
    for t in range(1, S):
        ids[:, t] = torch.where(follow[:, t], nxt[ids[:, t - 1]], ids[:, t])
    lens = torch.tensor(lengths)
    return ids.masked_fill(torch.arange(S)[None, :] >= lens[:, None], 0), lens


def _batch(case, cfg, seed):
    """A training batch: the first fifth of every sequence is its prompt."""
    ids, lens = _tokens(cfg, _lengths(case, case["sequences"]), seed)
    pos = torch.arange(ids.shape[1])[None, :]
    adv = torch.randn(len(lens), 1, generator=torch.Generator().manual_seed(seed + 1)).expand(ids.shape).contiguous()
    mask = ((pos >= lens[:, None] // 5) & (pos < lens[:, None])).float()
    batch = dict(input_ids=ids, input_lengths=lens, token_mask=mask, sample_mask=torch.ones(len(lens)), advantages=adv,
                 generation_logprobs=torch.zeros(ids.shape))
    if cfg.num_experts:
        g = torch.Generator("cuda").manual_seed(seed + 2)
        score = torch.rand((*ids.shape, cfg.num_hidden_layers, cfg.num_experts), device="cuda", generator=g)
        batch["routed_experts"] = score.topk(cfg.num_experts_per_tok, -1)[1].to(torch.int16).cpu()
    return batch


def prepare(case, seed):
    cfg = _config(case)
    if case["kind"] in ("generate", "prefill"):
        model = build_model(cfg, device="cuda", dtype=torch.bfloat16, init=False)
        _fill(model, case, cfg, seed)
        lengths, samples, new = _lengths(case, case["prompts"]), case.get("samples", 1), case.get("new_tokens", 1)
        ids, _ = _tokens(cfg, lengths, seed)
        prompts = [ids[i, :n].tolist() for i, n in enumerate(lengths) for _ in range(samples)]
        pages = sum(-(-n // BLOCK) + 1 for n in lengths) + len(prompts) * (-(-new // BLOCK) + 3)
        engine = GenerationEngine(model, block_size=BLOCK, num_blocks=pages + 16, max_running=max(8, len(prompts)),
                                  max_model_len=-(-(max(lengths) + new + 64) // 1024) * 1024)
        engine.wake()
        sp = SamplingParams(temperature=case.get("temperature") or 1.0, greedy=not case.get("temperature"), max_new_tokens=new, stop_token_ids=[], seed=seed % 1000)
        return dict(case=case, engine=engine, prompts=prompts, sampling=sp)
    budget = case["budget"]
    policy_cfg = dict(precision="bfloat16", train_global_batch_size=case["sequences"], train_micro_batch_size=case["sequences"],
                      logprob_batch_size=case["sequences"], max_total_sequence_length=2 * case["length"], max_grad_norm=MAX_NORM, grad_dtype="float32",
                      sequence_packing=dict(enabled=budget > 0, train_mb_tokens=budget, logprob_mb_tokens=budget),
                      optimizer=dict(name="torch.optim.AdamW", kwargs=dict(lr=LR, weight_decay=DECAY, betas=list(BETAS), eps=EPS)))
    if cfg.num_experts:
        policy_cfg["router_replay"] = dict(enabled=True)
    policy = PolicyWorker(policy_cfg, model_cfg=cfg, device="cuda", init_optimizer=case["kind"] == "train", init_reference_model=False)
    _fill(policy.model, case, cfg, seed)
    loss = NLLLossFn() if case.get("loss") == "sft" else ClippedPGLossFn(dict(force_on_policy_ratio=True, reference_policy_kl_penalty=0.0))
    return dict(case=case, policy=policy, data=BatchedDataDict(_batch(case, cfg, seed)), loss=loss)


# ------------------------------------------------------------------------------------------------------------------ runs
def run(state):
    case = state["case"]
    if case["kind"] == "generate":
        engine = state["engine"]
        done = engine.generate(state["prompts"], state["sampling"])
        engine.sleep(free_kv_cache=False)      # as a rollout phase ends
        return dict(tokens=torch.tensor([r.out_tokens for r in done]), logprobs=torch.tensor([r.out_logprobs for r in done]))
    if case["kind"] == "prefill":
        names = list(range(len(state["prompts"])))
        rows = state["engine"].step([(i, p, [len(p) - 1]) for i, p in zip(names, state["prompts"])], end=names)
        return dict(logits=torch.cat(rows))
    policy, data = state["policy"], state["data"]
    if case["kind"] == "logprobs":
        policy.prepare_for_lp_inference()
        return dict(logprobs=policy.get_logprobs(data)["logprobs"])
    policy.prepare_for_training()
    out = policy.train(data, state["loss"])
    return dict(loss=out["loss"], grad_norm=out["grad_norm"], weights=policy.flat.flat, momentum=policy.optimizer.m)


# ------------------------------------------------------------------------------------------------------------ what it costs
def _counts(cfg):
    """(parameters of the layers' products that one token goes through, all of the layers', of the output head, attention width)."""
    if cfg.is_mixer:
        att, ret = cfg.mixers[0]["mixer"], next(m["mixer"] for m in cfg.mixers if m["type"] == "retention")
        d, H = cfg.hidden_size, att["heads"]
        one = {"latent_attention": d * (H * (att["dim"] + att["rot_dim"] + 2 * att["vdim"]) + att["kv_rank"] + att["rot_dim"]) + att["kv_rank"] * H * (att["dim"] + att["vdim"]),
               "retention": d * ret["heads"] * (2 * ret["dim"] + 3 * ret["vdim"])}
        size = [one[m["type"]] + 2 * d * m["mlp"]["ff"] for m in cfg.mixers]
        attending = sum(cfg.mixers[i]["type"] == "latent_attention" for i, _ in cfg.layer_runs)
        return sum(size[i] for i, _ in cfg.layer_runs), sum(size), cfg.vocab_size * d, attending * H * (att["dim"] + att["rot_dim"] + att["vdim"])
    d, L = cfg.hidden_size, cfg.num_hidden_layers
    q, kv = cfg.num_attention_heads * cfg.head_dim, cfg.num_key_value_heads * cfg.head_dim
    attn = 2 * d * q + 2 * d * kv
    if cfg.num_experts:
        used, held = 3 * d * cfg.moe_intermediate_size * cfg.num_experts_per_tok + d * cfg.num_experts, (3 * d * cfg.moe_intermediate_size + d) * cfg.num_experts
    else:
        used = held = 3 * d * cfg.intermediate_size
    return L * (attn + used), L * (attn + held), cfg.vocab_size * d, 2 * L * q


def _cache_width(cfg):
    """Bytes that one token of context keeps."""
    if cfg.is_mixer:
        m = cfg.mixers[0]["mixer"]
        return 2 * (m["kv_rank"] + m["rot_dim"]) * sum(cfg.mixers[i]["type"] == "latent_attention" for i, _ in cfg.layer_runs)
    return 4 * cfg.num_hidden_layers * cfg.num_key_value_heads * cfg.head_dim


def work(case):
    cfg = _config(case)
    used, held, head, wide = _counts(cfg)
    if case["kind"] in ("generate", "prefill"):
        lengths, samples, steps = _lengths(case, case["prompts"]), case.get("samples", 1), case.get("new_tokens", 1) - 1
        n = len(lengths) * samples
        flops = sum(2 * used * t + wide * t * t for t in lengths) + 2 * head * len(lengths) + steps * n * 2 * (used + head) + steps * samples * 2 * wide * sum(lengths)
        experts = 1.0 if not cfg.num_experts else 1 - (1 - cfg.num_experts_per_tok / cfg.num_experts) ** n      # share of them that a step meets
        return dict(flops=flops, bytes=2 * (held + head) + steps * (2 * (held * experts + head) + _cache_width(cfg) * sum(lengths)))
    lengths = _lengths(case, case["sequences"])
    flops = sum(2 * (used + head) * t + wide * t * t for t in lengths)
    if case["kind"] == "logprobs":
        return dict(flops=flops, bytes=2 * (held + head) + 12 * sum(lengths))
    # weights twice, moments and master read and written, gradients written and read
    params = held + head * (1 if cfg.tie_word_embeddings else 2)
    return dict(flops=3 * flops, bytes=params * (2 * 2 + 2 * (4 + 4 + 4) + 2 * 4))


def tolerance(case):
    """Against float64 the bf16 paths are off by 2e-3 to 1e-2 in sampled tokens' log-probabilities, 1e-3 in those of given tokens, 2e-2 in the logits
    of 32 layers and 1e-2 in gradients; two such paths differ by as much. Single values: a gradient's smallest ones are sums of far larger terms."""
    if case["kind"] == "generate":
        return dict(rel=0.03, max=0.5, differ=0.01)
    return dict(rel=0.01 if case["kind"] == "logprobs" else 0.03, max=0.99 if case["kind"] == "train" else 0.5)


# --------------------------------------------------------------------------------------------------------------- in 64 bits
F64 = torch.float64


def _rms(x, w, eps):
    y = x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps)
    return y if w is None else y * w


def _frequencies(dims, base, scaling):
    """(angle per position of each rotated pair, factor on cosine and sine)."""
    f = base ** (-2.0 * torch.arange(dims // 2, dtype=F64, device="cuda") / dims)
    if not scaling:
        return f, 1.0
    turns = f / (2 * math.pi)
    if scaling.get("rope_type") == "llama3":
        old, lo, hi = scaling["original_max_position_embeddings"], scaling["low_freq_factor"], scaling["high_freq_factor"]
        keep = ((old * turns - lo) / (hi - lo)).clamp(0, 1)
        return keep * f + (1 - keep) * f / scaling["factor"], 1.0
    at = [dims * math.log(scaling["original"] / (2 * math.pi * t)) / (2 * math.log(base)) for t in (scaling["fast"], scaling["slow"])]
    lo, hi = max(math.floor(at[0]), 0), min(math.ceil(at[1]), dims - 1)
    slow = ((torch.arange(dims // 2, dtype=F64, device="cuda") - lo) / max(hi - lo, 1e-3)).clamp(0, 1)
    return f / scaling["factor"] * slow + f * (1 - slow), 0.1 * math.log(scaling["factor"]) + 1


def _rotate(x, positions, freq, gain=1.0, interleaved=False):
    """x [T, H, n], its leading 2 len(freq) entries rotated."""
    half = freq.numel()
    ang = positions.to(F64)[:, None] * freq
    c, s = (ang.cos() * gain)[:, None], (ang.sin() * gain)[:, None]
    h, rest = x[..., : 2 * half], x[..., 2 * half :]
    u, v = (h[..., 0::2], h[..., 1::2]) if interleaved else (h[..., :half], h[..., half:])
    a, b = u * c - v * s, v * c + u * s
    return torch.cat([torch.stack([a, b], -1).flatten(-2) if interleaved else torch.cat([a, b], -1), rest], -1)


def _attend(q, k, v, lengths, scale):
    """Causal attention of packed sequences, 1024 queries at a time; q [T, Hq, n], k and v with as many or fewer heads."""
    out, s = [], 0
    G = q.shape[1] // k.shape[1]
    for n in lengths:
        kh, vh = k[s : s + n].repeat_interleave(G, 1).transpose(0, 1), v[s : s + n].repeat_interleave(G, 1).transpose(0, 1)
        for a in range(0, n, 1024):
            b = min(n, a + 1024)
            z = q[s + a : s + b].transpose(0, 1) @ kh[:, :b].transpose(1, 2) * scale
            z = z.masked_fill(torch.arange(b, device=z.device)[None, :] > torch.arange(a, b, device=z.device)[:, None], -math.inf)
            out.append((torch.softmax(z, -1) @ vh[:, :b]).transpose(0, 1))
        s += n
    return torch.cat(out)


def _decoder64(cfg, W, ids, lengths, routed=None):
    """Normed final hidden states [T, d] of packed sequences; ``W(name)`` gives a weight in 64 bits, ``routed`` [T, layers, k] the experts."""
    H, Hk, D, eps = cfg.num_attention_heads, cfg.num_key_value_heads, cfg.head_dim, cfg.rms_norm_eps
    pos = torch.cat([torch.arange(n, device="cuda") for n in lengths])
    freq, _ = _frequencies(D, cfg.rope_theta, cfg.rope_scaling)
    h = W("embed_tokens")[ids]
    for i in range(cfg.num_hidden_layers):
        at = f"layers.{i}."
        qkv = (_rms(h, W(at + "input_layernorm"), eps) @ W(at + "self_attn.qkv_proj").T).view(len(ids), H + 2 * Hk, D)
        q, k, v = qkv[:, :H], qkv[:, H : H + Hk], qkv[:, H + Hk :]
        if cfg.qk_norm:
            q, k = _rms(q, W(at + "self_attn.q_norm"), eps), _rms(k, W(at + "self_attn.k_norm"), eps)
        a = _attend(_rotate(q, pos, freq), _rotate(k, pos, freq), v, lengths, D ** -0.5)
        h = h + a.reshape(len(ids), H * D) @ W(at + "self_attn.o_proj").T
        x = _rms(h, W(at + "post_attention_layernorm"), eps)
        up, down = W(at + "mlp.gate_up_proj"), W(at + "mlp.down_proj")
        if cfg.num_experts:
            p = torch.softmax(x @ W(at + "mlp.router").T, -1)
            chosen = p.topk(cfg.num_experts_per_tok, -1)[1] if routed is None else routed[:, i].long()
            p = p.gather(1, chosen)
            p = p / p.sum(-1, keepdim=True)
            for e in range(cfg.num_experts):
                t, j = (chosen == e).nonzero(as_tuple=True)
                if len(t):
                    g, u = (x[t] @ up[e].T).chunk(2, -1)
                    h = h.index_add(0, t, (torch.nn.functional.silu(g) * u) @ down[e].T * p[t, j, None])
        else:
            g, u = (x @ up.T).chunk(2, -1)
            h = h + (torch.nn.functional.silu(g) * u) @ down.T
    return _rms(h, W("norm"), eps)


def _layer_list64(cfg, W, ids, lengths):
    """The same of a layer-list model with parallel layers: latent attention or retention beside a squared-ReLU unit."""
    T, eps = len(ids), cfg.rms_norm_eps
    pos = torch.cat([torch.arange(n, device="cuda") for n in lengths])

    def norm(x, name):
        return torch.tanh(x * W(name + ".alpha")) * W(name + ".weight") + W(name + ".bias")

    e = W("embed_tokens")[ids] * cfg.embed_scale
    x, loop = e, cfg.layer_loop
    for i, again in cfg.layer_runs:
        if again is not None and i == loop["start"]:
            x = (x + e if again else x) + W("loop_step")[again]
        m, at = cfg.mixers[i]["mixer"], f"layers.{i}."
        H, dv = m["heads"], m["vdim"]
        h = norm(x, at + "norm")
        p = h @ W(at + "in_proj").T
        freq, gain = _frequencies(m["rot"]["dims"], m["rot"]["base"], m["rot"].get("scaling"))
        if cfg.mixers[i]["type"] == "latent_attention":
            n, r, R = m["dim"], m["rot_dim"], m["kv_rank"]
            q, lat, kr, gate, up = p.split([H * (n + r), R, r, H * dv, cfg.mixers[i]["mlp"]["ff"]], -1)
            q = q.view(T, H, n + r)
            kv = _rms(lat, W(at + "mixer.kv_norm"), eps) @ W(at + "mixer.kv_up").T
            q = torch.cat([q[..., :n], _rotate(q[..., n:], pos, freq, gain, True)], -1)
            k = torch.cat([kv[:, : H * n].view(T, H, n), _rotate(kr[:, None], pos, freq, gain, True).expand(T, H, r)], -1)
            y = _attend(q, k, kv[:, H * n :].view(T, H, dv), lengths, m["scale"]).reshape(T, H * dv) * torch.sigmoid(gate)
        else:
            n = m["dim"]
            q, k, v, gate, up = p.split([H * n, H * n, H * dv, H * dv, cfg.mixers[i]["mlp"]["ff"]], -1)
            q, k = _rotate(q.view(T, H, n), pos, freq), _rotate(k.view(T, H, n), pos, freq) * n ** -0.5
            fade = torch.tensor(m["decay"], dtype=F64, device="cuda").log()[:, None, None]
            parts, s = [], 0
            for t in lengths:
                gap = torch.arange(t, device="cuda")[:, None] - torch.arange(t, device="cuda")[None, :]
                w = torch.where(gap >= 0, torch.exp(gap.clamp(min=0) * fade), torch.zeros((), dtype=F64, device="cuda"))
                z = (q[s : s + t].transpose(0, 1) @ k[s : s + t].permute(1, 2, 0)) * w
                parts.append((z @ v[s : s + t].view(t, H, dv).transpose(0, 1)).transpose(0, 1))
                s += t
            y = _rms(torch.cat(parts), None, eps).reshape(T, H * dv) * torch.nn.functional.silu(gate)
        x = x + torch.cat([y, torch.relu(up).square()], -1) @ W(at + "out_proj").T
    return norm(x, "norm")


def _head_name(cfg):
    return "embed_tokens" if cfg.tie_word_embeddings else "lm_head"


def exact(case, seed):
    cfg, w = _config(case), work(case)
    if w["flops"] > EXACT_FLOPS or case.get("temperature"):
        return None
    shapes = {n: p.shape for n, p in build_model(cfg, device="meta", init=False).named_parameters()}

    def W(name):
        return _weight(case, cfg, name, shapes[name], seed).to(F64)

    hidden = _layer_list64 if cfg.is_mixer else _decoder64
    if case["kind"] == "train":
        return _train64(case, cfg, {n: W(n) for n in shapes}, seed)
    with torch.no_grad():
        if case["kind"] == "logprobs":
            data = _batch(case, cfg, seed)
            lens = data["input_lengths"].tolist()
            ids = torch.cat([data["input_ids"][i, :n] for i, n in enumerate(lens)]).cuda()
            h, head = hidden(cfg, W, ids, lens), W(_head_name(cfg))
            lp = torch.cat([torch.log_softmax(h[s : s + 1024] @ head.T, -1).gather(1, ids.roll(-1)[s : s + 1024, None])[:, 0] for s in range(0, len(ids), 1024)])
            out, s = torch.zeros(data["input_ids"].shape, dtype=F64, device="cuda"), 0
            for i, n in enumerate(lens):
                out[i, 1:n] = lp[s : s + n - 1]
                s += n
            return dict(logprobs=out)
        lengths, new = _lengths(case, case["prompts"]), case.get("new_tokens", 0)
        prompts, _ = _tokens(cfg, lengths, seed)
        head, nxt = W(_head_name(cfg)), _successor(cfg).cpu()
        if case["kind"] == "prefill":
            h = hidden(cfg, W, torch.cat([prompts[i, :n] for i, n in enumerate(lengths)]).cuda(), lengths)
            return dict(logits=h[torch.tensor(lengths).cumsum(0).cuda() - 1] @ head.T)
        rows = [prompts[i, :n].tolist() for i, n in enumerate(lengths)]

        def chain(row, upto):
            while len(row) < upto:
                row.append(int(nxt[row[-1]]))
            return row

        rows = [chain(r, n + new) for r, n in zip(rows, lengths)]
        for _ in range(4):      # the likely continuation, put right where the model says otherwise
            flat = torch.tensor([t for r in rows for t in r[:-1]], device="cuda")
            full = [n + new - 1 for n in lengths]
            h = hidden(cfg, W, flat, full)
            ends = torch.tensor(full).cumsum(0)
            at = torch.cat([torch.arange(e - new, e) for e in ends.tolist()]).cuda()
            lp = torch.log_softmax(h[at] @ head.T, -1)
            best, tok = lp.max(-1)
            tok = tok.view(len(rows), new).tolist()
            wrong = False
            for i, n in enumerate(lengths):
                j = next((j for j in range(new) if rows[i][n + j] != tok[i][j]), None)
                if j is not None:
                    rows[i], wrong = chain(rows[i][: n + j] + [tok[i][j]], n + new), True
            if not wrong:
                return dict(tokens=torch.tensor(tok), logprobs=best.view(len(rows), new))
    return None


def _train64(case, cfg, weights, seed):
    """Loss, clipped gradient and AdamW step, one sequence at a time."""
    data = _batch(case, cfg, seed)
    mask, adv = data["token_mask"].to(F64).cuda(), data["advantages"].to(F64).cuda()
    total, loss = mask[:, 1:].sum(), 0.0
    for p in weights.values():
        p.requires_grad_()
    for i, n in enumerate(data["input_lengths"].tolist()):
        ids = data["input_ids"][i, :n].cuda()
        h = _decoder64(cfg, weights.__getitem__, ids, [n], data["routed_experts"][i, :n].cuda() if cfg.num_experts else None)
        cut = h.detach().requires_grad_()
        for s in range(0, n - 1, 1024):
            e = min(n - 1, s + 1024)
            lp = torch.log_softmax(cut[s:e] @ weights[_head_name(cfg)].T, -1).gather(1, ids[s + 1 : e + 1, None])[:, 0]
            coef = mask[i, s + 1 : e + 1] if case["loss"] == "sft" else adv[i, s + 1 : e + 1] * mask[i, s + 1 : e + 1]
            part = -(coef * lp).sum() / total
            part.backward()
            # with a ratio of one the policy loss is minus the mean advantage; its gradient is that of the log-probabilities
            loss += float(part.detach()) if case["loss"] == "sft" else -float(coef.sum() / total)
        h.backward(cut.grad)
    with torch.no_grad():
        flat = lambda f: torch.cat([f(p).reshape(-1) for p in weights.values()])      # noqa: E731
        g = flat(lambda p: p.grad if p.grad is not None else torch.zeros_like(p))
        w = flat(lambda p: p)
        gn = g.norm()
        g *= min(1.0, MAX_NORM / (float(gn) + 1e-6))
        w = w * (1 - LR * DECAY) - LR * g / (g.abs() + EPS)      # the first step's bias corrections cancel the decays of the moments
        pad = -w.numel() % 256
        w, g = (torch.nn.functional.pad(t, (0, pad)) for t in (w, g * (1 - BETAS[0])))
    return dict(loss=torch.tensor([loss], dtype=F64), grad_norm=gn.reshape(1), weights=w, momentum=g)
