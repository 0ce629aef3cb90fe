"""Grouped GEMM and the MoE layer on a GPU against a plain fp32 per-expert reference."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref_mlp(xs, counts, gate_up, down):
    outs, s = [], 0
    for e, c in enumerate(counts):
        xe = xs[s : s + c].float()
        h = xe @ gate_up[e].float().t()
        f = h.shape[1] // 2
        a = torch.nn.functional.silu(h[:, :f]) * h[:, f:]
        outs.append(a.to(torch.bfloat16).float() @ down[e].float().t())
        s += c
    return torch.cat(outs, 0)


@pytest.mark.parametrize("counts", [[130, 0, 77, 256, 1, 0, 300, 5], [0, 0, 0, 64], [128, 128]])
def test_grouped_expert_mlp_forward_backward(native_lib, counts):
    from rl_b200.ops.lib import check_status
    from rl_b200.ops.moe_ops import grouped_expert_mlp

    torch.manual_seed(0)
    E, d, f = len(counts), 256, 192
    n = sum(counts)
    xs = (torch.randn(n, d, device="cuda") * 0.5).to(torch.bfloat16).requires_grad_(True)
    gu = (torch.randn(E, 2 * f, d, device="cuda") * 0.05).to(torch.bfloat16).requires_grad_(True)
    dn = (torch.randn(E, d, f, device="cuda") * 0.05).to(torch.bfloat16).requires_grad_(True)
    cnt = torch.tensor(counts, device="cuda")
    y = grouped_expert_mlp(xs, cnt, gu, dn)
    g = torch.randn_like(y)
    y.backward(g)
    torch.cuda.synchronize()
    assert check_status() == 0
    xr, gur, dnr = (t.detach().float().requires_grad_(True) for t in (xs, gu, dn))
    yr = _ref_mlp(xr, counts, gur, dnr)
    yr.backward(g.float())
    tol = lambda ref: 3e-2 * ref.abs().max().item() + 1e-3  # noqa: E731
    assert (y.float() - yr).abs().max().item() <= tol(yr)
    assert (xs.grad.float() - xr.grad).abs().max().item() <= tol(xr.grad)
    assert (gu.grad.float() - gur.grad).abs().max().item() <= tol(gur.grad)
    assert (dn.grad.float() - dnr.grad).abs().max().item() <= tol(dnr.grad)
    # experts without tokens get exactly zero weight gradient
    for e, c in enumerate(counts):
        if c == 0:
            assert gu.grad[e].abs().max().item() == 0 and dn.grad[e].abs().max().item() == 0


def test_moe_model_matches_fp32_reference(native_lib):
    from rl_b200.models.config import preset
    from rl_b200.models.transformer import PackedBatch, build_model
    from rl_b200.ops.lib import check_status

    cfg = preset("tiny-llama-oracle", num_experts=8, num_experts_per_tok=2, moe_intermediate_size=128, norm_topk_prob=True,
                 hidden_size=256, num_attention_heads=2, num_key_value_heads=1, head_dim=128, vocab_size=2048)
    from rl_b200.models.hf_io import iter_hf_tensors, load_hf_tensors

    m = build_model(cfg, device="cuda", dtype=torch.bfloat16, seed=5)
    ref = build_model(cfg, dtype=torch.float32, init=False)
    load_hf_tensors(ref, {n: t.detach().float().cpu() for n, t in iter_hf_tensors(m)}.get)  # same (bf16-rounded) weights
    ids = torch.randint(0, cfg.vocab_size, (3, 40))
    lens = torch.tensor([40, 25, 33])
    bc = PackedBatch.from_padded(ids, lens)
    bg = PackedBatch.from_padded(ids.cuda(), lens.cuda())
    bg.input_ids = bg.input_ids.to(torch.int32)
    lp, _ = m.next_token_logprobs(bg)
    lp.sum().backward()
    torch.cuda.synchronize()
    assert check_status() == 0
    # a freshly initialised router is nearly uniform, so bf16 rounding flips many top-k choices: the reference replays the
    # GPU model's routing and then has to agree on everything else
    for lg, lr in zip(m.layers, ref.layers):
        lr.mlp.forced_routing = lg.mlp.last_routing.cpu()
    with torch.no_grad():
        lp_ref, _ = ref.next_token_logprobs(bc)
    assert (lp.detach().cpu() - lp_ref).abs().max().item() < 0.06
    g = m.layers[0].mlp.gate_up_proj.grad
    assert g is not None and torch.isfinite(g).all() and g.abs().sum().item() > 0


def test_route_topk_kernel_matches_torch(native_lib):
    from rl_b200.ops.moe_ops import route_topk, route_topk_ref

    torch.manual_seed(0)
    for T, E, k, renorm in [(37, 128, 8, True), (5, 64, 2, False), (300, 8, 2, True), (64, 256, 16, True)]:
        z = (torch.randn(T, E, device="cuda") * 2).to(torch.bfloat16)
        w, idx = route_topk(z, k, renorm)
        w_ref, idx_ref = route_topk_ref(z, k, renorm)
        # equal probabilities (bf16 logits collide often) may be picked in another order: compare the weights, and the
        # experts through the probabilities they carry
        assert torch.allclose(w, w_ref, rtol=1e-4, atol=1e-6), (T, E, k)
        p = torch.softmax(z.float(), -1)
        assert torch.allclose(p.gather(1, idx.long()), p.gather(1, idx_ref.long()), rtol=1e-4, atol=1e-7)
        assert (idx.sort(1).values[:, 1:] != idx.sort(1).values[:, :-1]).all()     # k distinct experts per token


@pytest.mark.parametrize("T", [1, 48, 256])
def test_small_token_moe_layer_matches_sorted_path(native_lib, T):
    """The few-token layer (five kernels + two grouped GEMMs, no host visit) against the sort / scatter path of training."""
    from rl_b200.models.config import preset
    from rl_b200.models.moe import MoEMLP
    from rl_b200.ops.lib import check_status

    cfg = preset("tiny-llama-oracle", num_experts=16, num_experts_per_tok=4, moe_intermediate_size=128, norm_topk_prob=True, hidden_size=256)
    torch.manual_seed(1)
    m = MoEMLP(cfg, torch.bfloat16, "cuda")
    with torch.no_grad():
        m.router.copy_(torch.randn_like(m.router) * 0.5)
        m.gate_up_proj.copy_(torch.randn_like(m.gate_up_proj) * 0.06)
        m.down_proj.copy_(torch.randn_like(m.down_proj) * 0.06)
    x = torch.randn(T, 256, device="cuda").to(torch.bfloat16)
    res = torch.randn(T, 256, device="cuda").to(torch.bfloat16)
    with torch.no_grad():
        y_small = m(x, res)
        idx_small = m.last_routing.clone()
        assert m._small_workspace(T) is not None
    with torch.enable_grad():   # the training path (the few-token path is inference only)
        y_sorted = m(x, res).detach()
    torch.cuda.synchronize()
    assert check_status() == 0
    assert torch.equal(idx_small.long().sort(1).values, m.last_routing.long().sort(1).values)
    # fp32 statement with the same routing
    p = torch.softmax((x.float() @ m.router.float().t()).to(torch.bfloat16).float(), -1)
    w = p.gather(1, idx_small.long())
    w = w / w.sum(-1, keepdim=True)
    ref = res.float().clone()
    for t in range(T):
        for j in range(cfg.num_experts_per_tok):
            e = int(idx_small[t, j])
            h = x[t].float() @ m.gate_up_proj[e].float().t()
            a = (torch.nn.functional.silu(h[:128]) * h[128:]).to(torch.bfloat16).float()
            ref[t] += w[t, j] * (a @ m.down_proj[e].float().t())
    assert (y_small.float() - ref).abs().max().item() < 0.05, (y_small.float() - ref).abs().max().item()
    assert (y_small.float() - y_sorted.float()).abs().max().item() < 0.05


def test_moe_engine_decodes_from_cuda_graphs(native_lib):
    """A mixture-of-experts model decodes through captured graphs and produces the tokens of the step-by-step engine."""
    from rl_b200.engine.engine import GenerationEngine, SamplingParams
    from rl_b200.models.config import preset
    from rl_b200.models.transformer import build_model
    from rl_b200.ops.lib import check_status

    cfg = preset("tiny-llama-oracle", num_experts=8, num_experts_per_tok=2, moe_intermediate_size=128, norm_topk_prob=True,
                 hidden_size=256, num_attention_heads=2, num_key_value_heads=1, head_dim=128, vocab_size=2048)
    m = build_model(cfg, device="cuda", dtype=torch.bfloat16, seed=7)
    prompts = [[int(t) for t in torch.randint(1, 2048, (n,))] for n in (9, 17, 5, 30)]
    sp = SamplingParams(max_new_tokens=24, greedy=True)
    outs = {}
    for graphs in (True, False):
        eng = GenerationEngine(m, block_size=16, kv_cache_tokens=4096, max_running=8, use_cuda_graphs=graphs)
        outs[graphs] = [(r.out_tokens, r.out_logprobs) for r in eng.generate(prompts, sp)]
        if graphs:
            assert eng.use_graphs and len(eng._graphs) >= 1
    torch.cuda.synchronize()
    assert check_status() == 0
    same = sum(a[0] == b[0] for a, b in zip(outs[True], outs[False]))
    assert same >= 3, outs    # the same kernels run in both modes; a greedy near-tie may still split one sequence
    for a, b in zip(outs[True], outs[False]):
        if a[0] == b[0]:
            assert max(abs(x - y) for x, y in zip(a[1], b[1])) < 0.05


@pytest.mark.parametrize("T,E,k,skew", [(1, 8, 2, 0), (127, 128, 8, 0), (1300, 128, 8, 1), (700, 3, 1, 0), (2049, 256, 5, 2)])
@pytest.mark.parametrize("residual", [False, True])
def test_expert_layer(native_lib, T, E, k, skew, residual):
    """Plan, outputs and gradients of a whole layer: more than one block of copies, experts without tokens, one expert with most of them. Against
    float64 on the same bf16 values; every product's operands are bf16, so an output or gradient is off by a few roundings of 2^-9, relative to
    its norm: 1e-2."""
    from rl_b200.ops import moe_ops as M
    from rl_b200.ops.lib import check_status

    g = torch.Generator("cuda").manual_seed(T + E)
    d, f = 128, 64
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")      # noqa: E731
    score = r(T, E) + (torch.arange(E, device="cuda") == 1) * (5.0 if skew == 1 else 0.0) - (torch.arange(E, device="cuda") % 3 == 0) * (9.0 if skew == 2 else 0.0)
    idx = score.topk(k, -1)[1]
    plan = M.TokenPlan(idx, E)
    rows = plan.copy_row.long()
    counts = torch.bincount(idx.reshape(-1), minlength=E)
    assert torch.equal(plan.rows.long(), (counts + 127) // 128 * 128) and torch.equal(plan.row_copy[rows].long(), torch.arange(T * k, device="cuda"))
    assert torch.equal(plan.tile_expert[rows // 128].long(), idx.reshape(-1)) and (plan.row_copy >= 0).sum() == T * k
    order = torch.argsort(idx.reshape(-1), stable=True)      # rows of an expert hold its copies in order
    assert bool((rows[order][1:] > rows[order][:-1]).all())
    x, res = r(T, d).bfloat16().requires_grad_(), r(T, d).bfloat16().requires_grad_()
    w = torch.softmax(r(T, k), -1).requires_grad_()
    gu, dn = (0.2 * r(E, 2 * f, d)).bfloat16().requires_grad_(), (0.2 * r(E, d, f)).bfloat16().requires_grad_()
    dn.main_grad = torch.ones(E, d, f, device="cuda")
    dn2 = dn.detach().clone().requires_grad_()      # the same into a buffer whose old values are undefined; experts without tokens get zeros
    dn2.main_grad, dn2.grad_stale = torch.full((E, d, f), float("nan"), device="cuda"), True
    M.expert_layer(x.detach(), idx, w.detach(), None, gu.detach(), dn2).backward(torch.ones(T, d, device="cuda").bfloat16())
    assert not dn2.grad_stale and bool(torch.isfinite(dn2.main_grad).all()) and not bool(dn2.main_grad[counts == 0].any())
    out = M.expert_layer(x, idx, w, res if residual else None, gu, dn)
    up = r(T, d).bfloat16()
    out.backward(up)
    torch.cuda.synchronize()
    assert check_status() == 0
    X, R, W, G, D = (t.detach().double().requires_grad_() for t in (x, res, w, gu, dn))
    ref, size = R if residual else torch.zeros_like(R), torch.zeros_like(W)
    for e in range(E):
        t, j = (idx == e).nonzero(as_tuple=True)
        if len(t):
            a, b = (X[t] @ G[e].T).chunk(2, -1)
            y = (torch.nn.functional.silu(a) * b) @ D[e].T
            ref, size[t, j] = ref.index_add(0, t, y * W[t, j, None]), y.detach().norm(dim=-1)
    ref.backward(up.double())
    near = lambda a, b: (a.double() - b).norm() <= 1e-2 * b.norm() + 1e-12      # noqa: E731
    assert near(out, ref) and near(x.grad, X.grad) and near(gu.grad, G.grad) and near(dn.main_grad - 1, D.grad)
    # a weight's gradient is a scalar product whose terms may cancel: its error is relative to the factors' norms
    assert bool(((w.grad.double() - W.grad).abs() <= 1e-2 * up.double().norm(dim=-1, keepdim=True) * size.detach()).all())
    if residual:
        assert torch.equal(res.grad, up)
    assert gu.grad[counts == 0].abs().sum() == 0 and dn.grad is None


@pytest.mark.parametrize("what", ["tokens", "residual", "gradient"])
def test_expert_layer_rows_at_an_odd_place(native_lib, what):
    """Contiguous rows that do not start on 16 bytes are copied first: the same values as from aligned ones."""
    from rl_b200.ops import moe_ops as M
    from rl_b200.ops.lib import check_status

    g = torch.Generator("cuda").manual_seed(7)
    T, d, f, E, k = 40, 128, 64, 4, 2
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")      # noqa: E731
    x, res, up, w = r(T, d).bfloat16(), r(T, d).bfloat16(), r(T, d).bfloat16(), torch.softmax(r(T, k), -1)
    gu, dn, idx = (0.2 * r(E, 2 * f, d)).bfloat16(), (0.2 * r(E, d, f)).bfloat16(), r(T, E).topk(k, -1)[1]
    odd = lambda t: torch.cat([t.new_zeros(1), t.reshape(-1)])[1:].view(t.shape)      # noqa: E731

    def run(x, res, up):
        x, res = x.detach().requires_grad_(), res.detach().requires_grad_()
        y = M.expert_layer(x, idx, w, res, gu, dn)
        return [y, *torch.autograd.grad(y, (x, res), up)]

    plain = run(x, res, up)
    moved = run(odd(x) if what == "tokens" else x, odd(res) if what == "residual" else res, odd(up) if what == "gradient" else up)
    torch.cuda.synchronize()
    assert check_status() == 0 and all(torch.equal(a, b) for a, b in zip(plain, moved))


@pytest.mark.parametrize("T,E,k,load", [(1, 8, 2, 32), (33, 16, 4, 32), (126, 64, 8, 32), (60, 16, 6, 64), (64, 8, 4, 64), (128, 8, 4, 128)])
@pytest.mark.parametrize("one", [False, True])
def test_few_token_layer(native_lib, T, E, k, load, one):
    """Every tile size, experts without tokens, one expert with all of them (several tiles), widths that cut the last weight tile. Against float64:
    bf16 products, a unit rounded to bf16, weighted rows rounded to bf16: 1e-2 of the norm."""
    from rl_b200.ops import moe_ops as M
    from rl_b200.ops.lib import check_status

    g = torch.Generator("cuda").manual_seed(T + E)
    d, f = 192, 64
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")      # noqa: E731
    x, res, router = r(T, d).bfloat16(), r(T, d).bfloat16(), r(E, d).bfloat16()
    if one:
        x[:, 0], router[:, 0], router[1] = 100.0, 0, 0      # expert 1 scores 100, the others some 14 (sigma)
        router[1, 0] = 1.0
    gu, dn = (0.2 * r(E, 2 * f, d)).bfloat16(), (0.2 * r(E, d, f)).bfloat16()
    ws = M.SmallTokenMoE(d, f, E, k, None, T, x.device)
    assert ws.tile_rows(T) == load
    for _ in range(2):      # the workspace is used again
        out, idx = ws.forward(x, res, router, gu, dn, True)
    torch.cuda.synchronize()
    assert check_status() == 0
    W, ref = ws.w[:T].double(), res.double()
    for e in range(E):
        t, j = (idx == e).nonzero(as_tuple=True)
        if len(t):
            a, b = (x[t].double() @ gu[e].double().T).chunk(2, -1)
            ref = ref.index_add(0, t, (torch.nn.functional.silu(a) * b) @ dn[e].double().T * W[t, j, None])
    assert (out.double() - ref).norm() <= 1e-2 * ref.norm()
    if one:
        assert bool((idx == 1).any(-1).all())


@pytest.mark.parametrize("d,f", [(200, 64), (192, 72), (136, 40)])
def test_few_token_layer_widths(native_lib, d, f):
    """Widths that are not whole 64-column blocks take the grouped GEMM, as they did before there was another product. Bounds as above."""
    from rl_b200.ops import moe_ops as M
    from rl_b200.ops.lib import check_status

    T, E, k = 5, 8, 2
    g = torch.Generator("cuda").manual_seed(d)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")      # noqa: E731
    x, router = r(T, d).bfloat16(), r(E, d).bfloat16()
    gu, dn = (0.2 * r(E, 2 * f, d)).bfloat16(), (0.2 * r(E, d, f)).bfloat16()
    ws = M.SmallTokenMoE(d, f, E, k, None, T, x.device)
    out, idx = ws.forward(x, None, router, gu, dn, True)
    torch.cuda.synchronize()
    assert check_status() == 0
    ref = torch.zeros(T, d, dtype=torch.float64, device="cuda")
    for e in range(E):
        t, j = (idx == e).nonzero(as_tuple=True)
        if len(t):
            a, b = (x[t].double() @ gu[e].double().T).chunk(2, -1)
            ref = ref.index_add(0, t, (torch.nn.functional.silu(a) * b) @ dn[e].double().T * ws.w[:T].double()[t, j, None])
    assert (out.double() - ref).norm() <= 1e-2 * ref.norm()
