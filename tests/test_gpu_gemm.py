"""tcgen05 GEMM against an fp32 PyTorch matmul of the same bf16 operands, all three operand layouts,
ragged edges, accumulate / bias / fp32-output epilogues, and the fused lm_head log-prob epilogues."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel_err(a, b):
    return (a.float() - b.float()).abs().max().item() / (b.float().abs().max().item() + 1e-6)


SHAPES = [(128, 256, 64), (256, 512, 128), (300, 264, 200), (1000, 1024, 4096), (4096, 4096, 1024), (64, 8, 8)]


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("layout", ["kk", "k_mn", "mn_mn", "mn_k"])
def test_gemm_layouts(native_lib, M, N, K, layout):
    from rl_b200.ops import functional as F
    from rl_b200.ops.lib import check_status

    if layout != "kk" and (M % 8 or N % 8):
        pytest.skip("MN-major operands need 16-byte aligned rows")
    torch.manual_seed(0)
    dev = "cuda"
    a_mn = layout.startswith("mn")
    b_mn = layout.endswith("mn")
    a = torch.randn((K, M) if a_mn else (M, K), device=dev, dtype=torch.bfloat16)
    b = torch.randn((K, N) if b_mn else (N, K), device=dev, dtype=torch.bfloat16)
    ref = (a.t() if a_mn else a).float() @ (b if b_mn else b.t()).float()
    out = F.gemm(a, b, a_mn=a_mn, b_mn=b_mn)
    torch.cuda.synchronize()
    assert check_status() == 0
    assert _rel_err(out, ref) < 1e-2


def test_gemm_epilogues(native_lib):
    from rl_b200.ops import functional as F

    torch.manual_seed(1)
    M, N, K = 384, 520, 256
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(N, K, device="cuda", dtype=torch.bfloat16)
    bias = torch.randn(N, device="cuda")
    ref = a.float() @ b.float().t()
    out32 = F.gemm(a, b, out_dtype=torch.float32)
    assert _rel_err(out32, ref) < 2e-3
    outb = F.gemm(a, b, bias=bias)
    assert _rel_err(outb, ref + bias) < 1e-2
    acc = torch.ones(M, N, device="cuda", dtype=torch.float32)
    F.gemm(a, b, out=acc, accumulate=True)
    assert _rel_err(acc, ref + 1) < 2e-3
    accb = torch.ones(M, N, device="cuda", dtype=torch.bfloat16)
    F.gemm(a, b, out=accb, accumulate=True)
    assert _rel_err(accb, ref + 1) < 1e-2
    # strided views (slices of wider buffers)
    wide_a = torch.randn(M, K + 64, device="cuda", dtype=torch.bfloat16)
    wide_o = torch.zeros(M, N + 24, device="cuda", dtype=torch.bfloat16)
    F.gemm(wide_a[:, 64:], b, out=wide_o[:, 24:])
    assert _rel_err(wide_o[:, 24:], wide_a[:, 64:].float() @ b.float().t()) < 1e-2
    assert wide_o[:, :24].abs().max().item() == 0


@pytest.mark.parametrize("M", [8, 128, 136, 256, 264, 392])        # one CTA's rows of a 256-row tile, both CTAs', a ragged second tile
@pytest.mark.parametrize("N", [64, 72, 256, 328])                   # pieces of 64 columns, whole and cut; one tile and two
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_gemm_tile_edges(native_lib, M, N, dtype):
    """Accumulation, bias and residual at the edges of a pair's tile. Products of bf16 values are exact in fp32, so the fp32 result is off by
    the sums alone (K roundings of terms below 4 sigma^2: 1e-5 of the largest value); a bf16 result also by one
    rounding, at most 2^-8 of it (8 significant bits)."""
    from rl_b200.ops import functional as F
    from rl_b200.ops.lib import check_status

    torch.manual_seed(M + N)
    K = 456                                                         # seven k-blocks and an eighth that is cut: the ring wraps
    a, b = torch.randn(M, K, device="cuda", dtype=torch.bfloat16), torch.randn(N, K, device="cuda", dtype=torch.bfloat16)
    bias, res = torch.randn(N, device="cuda"), torch.randn(M, N, device="cuda", dtype=torch.bfloat16)
    wide = torch.randn(M + 1, N + 8, device="cuda").to(dtype)
    old = wide.clone()
    F.gemm(a, b, out=wide[:M, :N], bias=bias, residual=res, accumulate=True)
    ref = a.double() @ b.double().t() + bias + res + old[:M, :N]
    torch.cuda.synchronize()
    assert check_status() == 0
    bound = (1e-5 if dtype == torch.float32 else 2.0 ** -8 + 1e-5) * ref.abs().max()
    assert (wide[:M, :N].double() - ref).abs().max() <= bound
    assert torch.equal(wide[M:], old[M:]) and torch.equal(wide[:, N:], old[:, N:])      # nothing beside the tile is touched


@pytest.mark.parametrize("M,N,K,ctas", [(8, 72, 456, 1), (136, 328, 456, 1), (304, 584, 136, 1), (304, 584, 136, 3), (120, 20480, 128, 0), (1160, 4096, 72, 0)])
@pytest.mark.parametrize("layout", ["kk", "k_mn", "mn_mn", "mn_k"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_gemm_single_ctas(native_lib, M, N, K, ctas, layout, dtype):
    """One CTA a tile: asked for by the number of CTAs, or because it takes fewer waves than pairs (the last two sizes). Bounds as in test_gemm_tile_edges."""
    from rl_b200.ops import functional as F
    from rl_b200.ops.lib import check_status

    torch.manual_seed(M + N)
    a_mn, b_mn = layout.startswith("mn"), layout.endswith("mn")
    a, b = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(N, K, device="cuda").bfloat16()
    bias, res = torch.randn(N, device="cuda"), torch.randn(M, N, device="cuda").bfloat16()
    wide = torch.randn(M + 1, N + 8, device="cuda").to(dtype)
    old = wide.clone()
    F.gemm(a.t().contiguous() if a_mn else a, b.t().contiguous() if b_mn else b, a_mn=a_mn, b_mn=b_mn, out=wide[:M, :N], bias=bias, residual=res,
           accumulate=True, max_ctas=ctas)
    ref = a.double() @ b.double().t() + bias + res + old[:M, :N]
    torch.cuda.synchronize()
    assert check_status() == 0
    assert (wide[:M, :N].double() - ref).abs().max() <= (1e-5 if dtype == torch.float32 else 2.0 ** -8 + 1e-5) * ref.abs().max()
    assert torch.equal(wide[M:], old[M:]) and torch.equal(wide[:, N:], old[:, N:])


def test_linear_autograd(native_lib):
    from rl_b200.ops import functional as F

    torch.manual_seed(2)
    x = torch.randn(3, 100, 256, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    w = torch.randn(512, 256, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    y = F.linear(x, w)
    g = torch.randn_like(y)
    y.backward(g)
    xr = x.detach().float().requires_grad_()
    wr = w.detach().float().requires_grad_()
    yr = xr @ wr.t()
    yr.backward(g.float())
    assert _rel_err(y, yr) < 1e-2
    assert _rel_err(x.grad, xr.grad) < 1e-2
    assert _rel_err(w.grad, wr.grad) < 1e-2


@pytest.mark.parametrize("M,V,K", [(200, 1000, 128), (1024, 32000, 512), (77, 128256, 256)])
def test_lm_head_logprob(native_lib, M, V, K):
    from rl_b200.ops import functional as F
    from rl_b200.ops.lib import check_status

    torch.manual_seed(3)
    h = (torch.randn(M, K, device="cuda") * 0.5).to(torch.bfloat16).requires_grad_()
    w = (torch.randn(V, K, device="cuda") * 0.2).to(torch.bfloat16).requires_grad_()
    tg = torch.randint(0, V, (M,), device="cuda")
    temp = 0.8
    logp, ent = F.lm_head_logprobs(h, w, tg, temperature=temp, want_entropy=True)
    hr = h.detach().float().requires_grad_()
    wr = w.detach().float().requires_grad_()
    lr, er = F._lm_head_ref(hr, wr, tg, 1.0 / temp, True)
    assert check_status() == 0
    assert (logp - lr).abs().max().item() < 2e-2
    assert (ent - er).abs().max().item() < 2e-2
    cl = torch.randn(M, device="cuda")
    ce = torch.randn(M, device="cuda") * 0.1
    (logp * cl + ent * ce).sum().backward()
    (lr * cl + er * ce).sum().backward()
    assert _rel_err(h.grad, hr.grad) < 3e-2
    assert _rel_err(w.grad, wr.grad) < 3e-2


@pytest.mark.parametrize("M,V", [(1, 8), (33, 264), (129, 4096), (300, 4104), (257, 6152)])
def test_lm_head_kept_logits(native_lib, monkeypatch, M, V):
    """Gradients from the logits that forward kept (whole and partial runs of 4096 columns, last pieces of 8 and 32, rows in chunks) against
    float64, and those of the recomputed product. dZ is rounded to bf16 (2^-9 a value), dH once more: below 2^-8 of the norm."""
    from rl_b200.ops import functional as F

    K = 192
    g = torch.Generator("cuda").manual_seed(M)
    h = (torch.randn(M, K, generator=g, device="cuda") * 0.5).bfloat16()
    w = (torch.randn(V, K, generator=g, device="cuda") * 0.2).bfloat16()
    tg = torch.randint(0, V, (M,), generator=g, device="cuda")
    cl, ce = torch.randn(M, generator=g, device="cuda"), torch.randn(M, generator=g, device="cuda") * 0.1
    monkeypatch.setattr(F._LMHeadLogprob, "CHUNK", 128)
    kept = F._kept_logits
    calls = []
    grads = []
    for keep in (True, False):
        monkeypatch.setattr(F, "_kept_logits", lambda *a: (calls.append(a), kept(*a))[1] if keep else None)
        hg, wg = h.clone().requires_grad_(), w.clone().requires_grad_()
        lp, ent = F.lm_head_logprobs(hg, wg, tg, temperature=0.8, want_entropy=True)
        (lp * cl + ent * ce).sum().backward()
        grads.append((hg.grad, wg.grad))
    assert len(calls) == 1
    hd, wd = h.double().requires_grad_(), w.double().requires_grad_()
    logp = torch.log_softmax(hd @ wd.t() / 0.8, -1)
    (logp.gather(1, tg[:, None])[:, 0] * cl - (logp.exp() * logp).sum(-1) * ce).sum().backward()
    for got in grads:
        for x, ref in zip(got, (hd.grad, wd.grad)):
            assert (x.double() - ref).norm() <= 2.0 ** -8 * ref.norm()


@pytest.mark.parametrize("M,V", [(1, 8), (33, 264), (129, 4096), (300, 4104), (257, 6152)])
def test_lm_head_kept_logits_are_those_of_the_product(native_lib, monkeypatch, M, V):
    """Storage is given whatever the device has free, so that the kept logits are written and read; the values behind the last row and the gradients are
    looked at. Both ways start from the same scaled fp32 logits: dZ differs where one exponential lies on the other side of a rounding, 2^-8 of
    a value, a few in a thousand."""
    from rl_b200.ops import functional as F

    g = torch.Generator("cuda").manual_seed(M)
    h = (torch.randn(M, 192, generator=g, device="cuda") * 0.5).bfloat16()
    w = (torch.randn(V, 192, generator=g, device="cuda") * 0.2).bfloat16()
    tg = torch.randint(0, V, (M,), generator=g, device="cuda")
    cl, ce = torch.randn(M, generator=g, device="cuda"), torch.randn(M, generator=g, device="cuda") * 0.1
    monkeypatch.setattr(F._LMHeadLogprob, "CHUNK", 128)
    room = torch.full((M + 3, V), float("nan"), device="cuda")
    grads = []
    for z in (room, None):
        monkeypatch.setattr(F, "_kept_logits", lambda *a: z)
        hg, wg = h.clone().requires_grad_(), w.clone().requires_grad_()
        lp, ent = F.lm_head_logprobs(hg, wg, tg, temperature=0.8, want_entropy=True)
        (lp * cl + ent * ce).sum().backward()
        grads.append((hg.grad.double(), wg.grad.double()))
    want = h.double() @ w.double().t() / 0.8
    assert (room[:M].double() - want).abs().max() <= 1e-5 * want.abs().max() and bool(room[M:].isnan().all())
    for kept, again in zip(*grads):
        assert (kept - again).norm() <= 2.0 ** -9 * again.norm()


@pytest.mark.parametrize("T", [0, 1, 130, 700])
def test_stale_gradients_are_written_over(native_lib, monkeypatch, T):
    """Gradients of a linear layer (used once and twice), of the vocabulary product in chunks and of an embedding into buffers whose old values are
    undefined, equal to those added to zeros: x + 0 is x."""
    from rl_b200.ops import functional as F

    monkeypatch.setattr(F._LMHeadLogprob, "CHUNK", 64)
    g = torch.Generator("cuda").manual_seed(T)
    rnd = lambda *s: (torch.randn(*s, generator=g, device="cuda") * 0.1).bfloat16()      # noqa: E731
    ids = torch.randint(0, 136, (T,), generator=g, device="cuda")
    shapes = dict(once=(264, 128), twice=(128, 128), head=(136, 128), table=(136, 128))
    weights = {n: rnd(*s) for n, s in shapes.items()}
    x, up = rnd(T, 128), rnd(T, 264)
    grads = []
    for stale in (False, True):
        ps = {n: torch.nn.Parameter(w.clone()) for n, w in weights.items()}
        for p in ps.values():
            p.main_grad = torch.full(p.shape, float("nan") if stale else 0.0, device="cuda")
            p.grad_stale = stale
        h = F.embedding(ids, ps["table"]) + x
        h = F.linear(F.linear(h, ps["twice"]), ps["twice"])
        loss = (F.linear(h, ps["once"]) * up).sum()
        if T:
            loss = loss + F.lm_head_logprobs(h, ps["head"], ids)[0].sum()
        loss.backward()
        grads.append({n: F.grad_buffer(p) for n, p in ps.items()})
    for n in shapes:
        assert torch.equal(grads[0][n], grads[1][n]) if n != "table" else torch.allclose(grads[0][n], grads[1][n], rtol=1e-4, atol=1e-6)


@pytest.mark.parametrize("parts", [1, 3, 8, 21])
def test_logprob_combine_empty_parts(native_lib, parts):
    """Parts without columns (maximum -inf, sums 0), as many as all of a warp's, count for nothing. Against float64: fp32 sums of at most 21 terms
    and the fast exponentials, 1e-5."""
    from rl_b200.ops.lib import call, ptr, stream_ptr

    M = 70
    g = torch.Generator("cuda").manual_seed(parts)
    mx, sm = torch.randn(parts, M, generator=g, device="cuda"), 1 + 50 * torch.rand(parts, M, generator=g, device="cuda")
    zs, tl = sm * torch.randn(parts, M, generator=g, device="cuda"), torch.randn(M, generator=g, device="cuda")
    empty = torch.rand(parts, M, generator=g, device="cuda") < 0.5
    empty[torch.randint(0, parts, (M,), generator=g, device="cuda"), torch.arange(M, device="cuda")] = False
    mx[empty], sm[empty], zs[empty] = -float("inf"), 0.0, 0.0
    lp, ent, lse = torch.empty(3, M, device="cuda")
    call("rlb_logprob_combine", ptr(mx), ptr(sm), ptr(zs), ptr(tl), M, parts, ptr(lp), ptr(ent), ptr(lse), stream_ptr())
    w = torch.exp(mx.double())
    total = (w * sm).sum(0)
    for got, ref in ((lse, total.log()), (lp, tl - total.log()), (ent, total.log() - (w * zs).sum(0) / total)):
        assert (got - ref).abs().max() <= 1e-5 * (1 + ref.abs().max())


@pytest.mark.parametrize("M", [1, 7, 32, 64, 100, 128, 200, 256])
@pytest.mark.parametrize("N,K", [(4096, 4096), (6144, 4096), (4096, 14336), (1000, 512), (128256, 1024)])
def test_skinny_gemm(native_lib, M, N, K):
    """Decode-sized GEMM (operands swapped, cluster split-K) against fp32 matmul, with bias / residual / fp32 output."""
    from rl_b200.ops import functional as F
    from rl_b200.ops.lib import check_status

    torch.manual_seed(M + N)
    x = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    w = (torch.randn(N, K, device="cuda") * 0.05).to(torch.bfloat16)
    ref = x.float() @ w.float().t()
    y = F.gemm(x, w)
    torch.cuda.synchronize()
    assert check_status() == 0
    assert _rel_err(y, ref) < 1e-2
    res = torch.randn(M, N, device="cuda", dtype=torch.bfloat16)
    bias = torch.randn(N, device="cuda")
    y2 = F.gemm(x, w, bias=bias, residual=res, out_dtype=torch.float32)
    assert _rel_err(y2, ref + bias + res.float()) < 2e-3


@pytest.mark.parametrize("M", [5, 128, 129, 256])
@pytest.mark.parametrize("N,K", [(19072, 512), (18952, 264), (9480, 448), (264, 256), (1000, 2048)])      # too wide to be split, contractions too short, split
@pytest.mark.parametrize("place", ["residual stride", "residual", "output", "both"])
def test_gemm_of_places_on_8_bytes(native_lib, M, N, K, place):
    """Up to 256 rows a residual's rows may be a multiple of four elements apart, and it and a bf16 output may start on 8 bytes. Against float64: fp32
    sums and one bf16 rounding of at most 2^-8, and not a value beside the output is written. 257 rows of such a residual are refused, and so is an
    fp32 output on 8 bytes, whatever the number of rows."""
    from rl_b200.ops import functional as F
    from rl_b200.ops.lib import NativeLibraryError, check_status

    g = torch.Generator("cuda").manual_seed(M + N)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")      # noqa: E731
    a, b = r(M, K).bfloat16(), (0.1 * r(N, K)).bfloat16()
    res = r(M, N + 4).bfloat16()[:, :N] if place == "residual stride" else r(M, N + 8).bfloat16()[:, 0 if place == "output" else 4 :][:, :N]
    wide = r(M, N + 8).bfloat16()
    old, at = wide.clone(), 4 if place in ("output", "both") else 0
    F.gemm(a, b, out=wide[:, at : at + N], residual=res)
    ref = a.double() @ b.double().t() + res
    torch.cuda.synchronize()
    assert check_status() == 0
    assert (wide[:, at : at + N].double() - ref).abs().max() <= (2.0 ** -8 + 1e-5) * ref.abs().max()
    assert torch.equal(wide[:, :at], old[:, :at]) and torch.equal(wide[:, at + N :], old[:, at + N :])
    with pytest.raises(NativeLibraryError):
        F.gemm(a, b, out=r(M, N + 4)[:, 2 : 2 + N])
    with pytest.raises(NativeLibraryError):
        F.gemm(r(257, K).bfloat16(), b, residual=r(257, N + 4).bfloat16()[:, :N])


@pytest.mark.parametrize("M", [129, 200, 256])
@pytest.mark.parametrize("N,K", [(3072, 2048), (6144, 4096), (4096, 14336), (16384, 2048), (16384, 576), (2048, 4992), (264, 520)])      # split by 8, 4, 2; halves of odd lengths
@pytest.mark.parametrize("kind", ["plain", "unit", "layer"])
def test_products_of_two_token_tiles_are_as_exact(native_lib, M, N, K, kind):
    """Sums over the contraction lose with their length. A product of 129 to 256 rows is cut into the same lengths as one of 128: its error against
    float64 is that of its first 128 rows (which differ by the chance of their values, some per cent; sums twice as long are off by twice as much)."""
    from rl_b200.ops import engine_ops as E
    from rl_b200.ops import functional as F
    from rl_b200.ops import layer_ops as Y
    from rl_b200.ops.lib import check_status

    g = torch.Generator("cuda").manual_seed(M + N)
    x, w = torch.randn(M, K, generator=g, device="cuda").bfloat16(), (0.05 * torch.randn(N, K, generator=g, device="cuda")).bfloat16()
    z = x.double() @ w.double().t()
    if kind == "unit":
        if N % 128:
            pytest.skip("the unit's halves are whole tiles")
        run = lambda t: E.skinny_linear(t, w, out_dtype=torch.float32, swiglu=True)      # noqa: E731
        z = torch.nn.functional.silu(z[:, : N // 2]) * z[:, N // 2 :]
    elif kind == "layer":
        run = lambda t: Y.capped_logits(t, w, 1.0, 0.0)      # noqa: E731
    else:
        run = lambda t: F.gemm(t, w, out_dtype=torch.float32)      # noqa: E731
    err = [((run(x[:m]) - z[:m]).norm() / z[:m].norm()).item() for m in (128, M)]
    assert check_status() == 0
    assert err[1] <= 1.2 * err[0] and err[0] < 1e-5


@pytest.mark.parametrize("M", [129, 130, 255, 257, 384, 385, 512, 640, 1000, 1024])      # token tiles of 128, whole and cut
@pytest.mark.parametrize("N,K", [(1000, 512), (2048, 264), (264, 8192), (4096, 1024)])
def test_skinny_token_tiles(native_lib, M, N, K):
    """More tokens than one tile holds, with norm statistics from and for the neighbours, against fp32. Inputs of one: a bf16 result is off by 2^-9
    of itself, the sums of its squares by fp32 rounding and that."""
    from rl_b200.ops import engine_ops as E
    from rl_b200.ops.lib import call, check_status, lib, ptr, status_word, stream_ptr

    g = torch.Generator("cuda").manual_seed(M + N)
    x, w = torch.randn(M, K, generator=g, device="cuda").bfloat16(), (torch.randn(N, K, generator=g, device="cuda") / K ** 0.5).bfloat16()
    res, bias = torch.randn(M, N, generator=g, device="cuda").bfloat16(), torch.randn(N, generator=g, device="cuda")
    ref = x.float() @ w.float().t() + bias + res.float()
    for split in (0, 1, 3, 8):
        y = torch.full((M + 1, N), 7.0, device="cuda").bfloat16()
        call("rlb_gemm_skinny", ptr(x), ptr(w), ptr(y), M, N, K, K, K, N, 0, ptr(bias), ptr(res), N, split, ptr(status_word(x.device)), stream_ptr())
        assert (y[:M].float() - ref).abs().max() <= 2.0 ** -8 * ref.abs().max() and bool((y[M] == 7).all())
    assert check_status() == 0
    if N % 128 == 0 and M <= 256:      # the decode step's hand-off of norm statistics
        ssq, hw, nw = torch.zeros(N // 128, 256, device="cuda"), torch.empty(M, N, device="cuda").bfloat16(), torch.rand(N, generator=g, device="cuda").bfloat16()
        h = E.skinny_linear(x, w, residual=res, ssq_out=ssq, norm_w=nw, out2=hw)
        assert torch.allclose(ssq[:, :M].sum(0), h.float().pow(2).sum(1), rtol=1e-4)
        assert (hw.float() - h.float() * nw.float()).abs().max() <= 2.0 ** -8 * h.float().abs().max()
        w2 = (torch.randn(256, N, generator=g, device="cuda") / N ** 0.5).bfloat16()
        act = E.skinny_linear(hw, w2, ssq_in=ssq, eps=1e-5, swiglu=True)
        z = (hw.float() @ w2.float().t()) * torch.rsqrt(h.float().pow(2).mean(1, keepdim=True) + 1e-5)
        want = torch.nn.functional.silu(z[:, :128]) * z[:, 128:]
        assert (act.float() - want).abs().max() <= 2.0 ** -7 * want.abs().max()


def test_skinny_split_values(native_lib):
    from rl_b200.ops.lib import call, lib, ptr, status_word, stream_ptr

    x = torch.randn(64, 4096, device="cuda", dtype=torch.bfloat16)
    w = (torch.randn(4096, 4096, device="cuda") * 0.05).to(torch.bfloat16)
    ref = x.float() @ w.float().t()
    outs = []
    for split in (1, 2, 3, 4, 8):
        y = torch.empty(64, 4096, device="cuda", dtype=torch.bfloat16)
        call("rlb_gemm_skinny", ptr(x), ptr(w), ptr(y), 64, 4096, 4096, 4096, 4096, 4096, 0, None, None, 0, split,
             ptr(status_word()), stream_ptr())
        assert _rel_err(y, ref) < 1e-2, split
        outs.append(y)
    assert lib().rlb_gemm_skinny_split(4096, 4096) in (1, 2, 4, 8)


@pytest.mark.parametrize("M", [1, 33, 65, 130])      # rings of four, four and three stages, two token tiles
@pytest.mark.parametrize("K", [64, 192, 256, 264, 320, 576, 1088])
@pytest.mark.parametrize("split", [1, 2, 4, 8])
def test_skinny_early_weights(native_lib, M, K, split):
    """Weights requested ahead of the dependency: ranges shorter than the ring, as long, longer and empty (more CTAs than blocks of 64). The same
    products in the same order as without, so equal bit for bit; against float64 one bf16 rounding and fp32 sums."""
    from rl_b200.ops.engine_ops import skinny_static_weights
    from rl_b200.ops.lib import call, check_status, ptr, status_word, stream_ptr

    g = torch.Generator("cuda").manual_seed(K + M)
    x, w = torch.randn(M, K, generator=g, device="cuda").bfloat16(), torch.randn(384, K, generator=g, device="cuda").bfloat16()
    outs = []
    for on in (False, True):
        y = torch.empty(M, 384, device="cuda", dtype=torch.bfloat16)
        torch.cuda.synchronize()      # (the promise holds: nothing writes the weights behind this)
        before = skinny_static_weights(on)
        for _ in range(3):
            call("rlb_gemm_skinny", ptr(x), ptr(w), ptr(y), M, 384, K, K, K, 384, 0, None, None, 0, split, ptr(status_word()), stream_ptr())
        skinny_static_weights(bool(before))
        outs.append(y)
    ref = x.double() @ w.double().t()
    assert check_status() == 0 and torch.equal(*outs)
    assert (outs[0].double() - ref).abs().max() <= (2.0 ** -8 + 1e-5) * ref.abs().max()


@pytest.mark.parametrize("M", [5, 64, 130])
def test_skinny_gemm_epilogue_fusions_match_fp32_reference(native_lib, M):
    """RMSNorm folded into two projections (producer writes h * w and per-tile sums of squares, consumer scales its rows)
    and SwiGLU in the gate_up epilogue, against the fp32 statement of norm -> linear -> swiglu -> linear."""
    from rl_b200.ops.engine_ops import skinny_linear
    from rl_b200.ops.lib import check_status

    torch.manual_seed(M)
    d, f, eps = 512, 1408, 1e-5
    dev = "cuda"
    a = torch.randn(M, d, device=dev).to(torch.bfloat16)
    res = torch.randn(M, d, device=dev).to(torch.bfloat16)
    w_o = (torch.randn(d, d, device=dev) / d**0.5).to(torch.bfloat16)
    w_norm = (1 + 0.1 * torch.randn(d, device=dev)).to(torch.bfloat16)
    w_gu = (torch.randn(2 * f, d, device=dev) / d**0.5).to(torch.bfloat16)
    w_dn = (torch.randn(d, f, device=dev) / f**0.5).to(torch.bfloat16)
    tiles = d // 128
    ssq = torch.zeros((tiles, 256), device=dev)
    hw = torch.empty((M, d), device=dev, dtype=torch.bfloat16)
    # producer: h = a W_o^T + res, plus h * w_norm and the per-tile sums of squares
    h = skinny_linear(a, w_o, residual=res, ssq_out=ssq, norm_w=w_norm, out2=hw)
    h_ref = (a.float() @ w_o.float().t() + res.float())
    assert (h.float() - h_ref).abs().max().item() < 3e-2 * h_ref.abs().max().item()
    hb = h.float()
    assert torch.allclose(ssq[:, :M].sum(0), (hb * hb).sum(-1), rtol=1e-4)
    assert (hw.float() - hb * w_norm.float()).abs().max().item() < 2e-2 * hb.abs().max().item()
    # consumer with SwiGLU: silu(norm(h) Wg^T) * (norm(h) Wu^T)
    act = skinny_linear(hw, w_gu, ssq_in=ssq, eps=eps, swiglu=True)
    xn = hb * torch.rsqrt((hb * hb).mean(-1, keepdim=True) + eps) * w_norm.float()
    gu = xn @ w_gu.float().t()
    act_ref = torch.nn.functional.silu(gu[:, :f]) * gu[:, f:]
    assert act.shape == (M, f)
    assert (act.float() - act_ref).abs().max().item() < 3e-2 * act_ref.abs().max().item() + 1e-3
    # consumer without SwiGLU, fp32 output and a bias (lm_head / qkv form)
    bias = torch.randn(d, device=dev)
    y = skinny_linear(hw, w_o, ssq_in=ssq, eps=eps, bias=bias, out_dtype=torch.float32)
    y_ref = xn @ w_o.float().t() + bias
    assert (y - y_ref).abs().max().item() < 2e-2 * y_ref.abs().max().item()
    # and the down projection closes the loop with the next norm's hand-off
    h2 = skinny_linear(act, w_dn, residual=h, ssq_out=ssq, norm_w=w_norm, out2=hw)
    h2_ref = act.float() @ w_dn.float().t() + hb
    assert (h2.float() - h2_ref).abs().max().item() < 3e-2 * h2_ref.abs().max().item()
    assert check_status() == 0
