"""tcgen05 flash attention (varlen, causal, GQA) against fp32 PyTorch attention, forward and backward."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(lens, Hq, Hkv, seed=0, D=128):
    torch.manual_seed(seed)
    T = sum(lens)
    qkv = (torch.randn(T, (Hq + 2 * Hkv) * D, device="cuda") * 0.7).to(torch.bfloat16)
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device="cuda")
    return qkv, cu, D


@pytest.mark.parametrize("D", [128, 64])
@pytest.mark.parametrize("lens,Hq,Hkv", [([128], 2, 2), ([64], 4, 1), ([200, 57, 1, 333], 8, 2), ([1280] * 3, 32, 8), ([4096], 4, 4)])
def test_flash_fwd(native_lib, lens, Hq, Hkv, D):
    from rl_b200.ops import attention as A
    from rl_b200.ops import functional as F
    from rl_b200.ops.lib import check_status

    qkv, cu, D = _case(lens, Hq, Hkv, D=D)
    out, lse = A.flash_fwd(qkv, cu, Hq, Hkv, D, 1.0 / math.sqrt(D))
    torch.cuda.synchronize()
    assert check_status() == 0
    ref = F._attention_ref(qkv.float(), cu, Hq, Hkv, D, 1.0 / math.sqrt(D))
    err = (out.float() - ref).abs().max().item()
    assert err < 3e-2, f"max abs err {err}"
    # lse against the direct definition on the first sequence / head 0
    n = lens[0]
    q = qkv[:n, :D].float()
    k = qkv[:n, Hq * D : Hq * D + D].float()
    s = (q @ k.t()) / math.sqrt(D)
    s = s.masked_fill(torch.triu(torch.ones(n, n, device="cuda", dtype=torch.bool), 1), float("-inf"))
    assert (torch.logsumexp(s, -1) - lse[0, :n]).abs().max().item() < 2e-2


@pytest.mark.parametrize("D", [128, 64])
@pytest.mark.parametrize("lens,Hq,Hkv", [([128], 2, 2), ([200, 57, 1, 333], 8, 2), ([1280, 700], 8, 2)])
def test_flash_autograd(native_lib, lens, Hq, Hkv, D):
    from rl_b200.ops import functional as F
    from rl_b200.ops.lib import check_status

    qkv, cu, D = _case(lens, Hq, Hkv, seed=1, D=D)
    x = qkv.clone().requires_grad_()
    y = F.attention_varlen(x, cu, max(lens), Hq, Hkv, D)
    g = torch.randn_like(y)
    y.backward(g)
    torch.cuda.synchronize()
    assert check_status() == 0
    xr = qkv.float().requires_grad_()
    yr = F._attention_ref(xr, cu, Hq, Hkv, D, 1.0 / math.sqrt(D))
    yr.backward(g.float())
    assert (y.float() - yr).abs().max().item() < 3e-2
    rel = (x.grad.float() - xr.grad).abs().max().item() / (xr.grad.abs().max().item() + 1e-6)
    assert rel < 3e-2, f"relative grad err {rel}"


@pytest.mark.parametrize("D", [128, 64])
@pytest.mark.parametrize("Hq,Hkv", [(2, 2), (3, 1), (8, 2)])
@pytest.mark.parametrize("n", [65, 129, 160, 192, 193, 257, 320, 321])
def test_flash_bwd_few_tiles(native_lib, n, Hq, Hkv, D):
    """Gradients where a tile has one to six tiles opposite it, both parities, next to a sequence of another length. Bound: that of test_flash_autograd.
    Nothing is summed by atomics, so repeats are equal bit for bit."""
    from rl_b200.ops import functional as F
    from rl_b200.ops.lib import check_status

    lens = [n, 70, n]
    qkv, cu, D = _case(lens, Hq, Hkv, seed=n, D=D)
    x = qkv.clone().requires_grad_()
    y = F.attention_varlen(x, cu, n, Hq, Hkv, D)
    g = torch.randn_like(y)
    grads = [torch.autograd.grad(y, x, g, retain_graph=True)[0] for _ in range(100)]
    torch.cuda.synchronize()
    assert check_status() == 0 and all(torch.equal(t, grads[0]) for t in grads[1:])
    xr = qkv.float().requires_grad_()
    F._attention_ref(xr, cu, Hq, Hkv, D, 1.0 / math.sqrt(D)).backward(g.float())
    assert (grads[0].float() - xr.grad).abs().max() <= 3e-2 * xr.grad.abs().max()


@pytest.mark.parametrize("D", [128, 64])
@pytest.mark.parametrize("n", [384, 385, 512, 513, 770])
def test_flash_bwd_more_tiles(native_lib, n, D):
    """The same with three to seven tiles of 128 opposite a tile: every slot of the rings and both places of the scores come round again."""
    test_flash_bwd_few_tiles(native_lib, n, 3, 1, D)


@pytest.mark.parametrize("D", [128, 64])
@pytest.mark.parametrize("scale", [0.0, -0.0, 1e-39, -1e-39, -0.09, 1e-3])
def test_flash_fwd_scales(native_lib, D, scale):
    """Scales of zero, too small for a normal number, and negative ones, where the least score has the largest weight. Bounds of test_flash_fwd."""
    from rl_b200.ops import attention as A
    from rl_b200.ops import functional as F
    from rl_b200.ops.lib import check_status

    qkv, cu, D = _case([200, 1, 333], 4, 2, seed=3, D=D)
    out, lse = A.flash_fwd(qkv, cu, 4, 2, D, scale)
    torch.cuda.synchronize()
    assert check_status() == 0 and bool(lse.isfinite().all())
    ref = F._attention_ref(qkv.float(), cu, 4, 2, D, scale)
    assert (out.float() - ref).abs().max() < 3e-2


@pytest.mark.parametrize("D", [128, 64])
@pytest.mark.parametrize("lens", [[300] * 3, [1, 640, 129, 128, 640, 0, 257], [33] * 128, [150, 20] * 64 + [40], [2000] + [10] * 20, [200] * 140])
def test_flash_tiles_of_every_sequence(native_lib, lens, D):
    """Equal lengths, all levels of work with several sequences in each, as many sequences as are sorted and one more, and enough tiles for the
    forward pass to go head by head: outputs and gradients of the longest and the shortest row of each, within the bf16 bounds above."""
    from rl_b200.ops import functional as F
    from rl_b200.ops.lib import check_status

    Hq, Hkv = (32, 4) if len(lens) == 140 else (4, 2)
    qkv, cu, D = _case(lens, Hq, Hkv, seed=len(lens), D=D)
    x = qkv.clone().requires_grad_()
    y = F.attention_varlen(x, cu, max(lens), Hq, Hkv, D)
    g = torch.randn_like(y)
    y.backward(g)
    torch.cuda.synchronize()
    assert check_status() == 0
    xr = qkv.float().requires_grad_()
    yr = F._attention_ref(xr, cu, Hq, Hkv, D, 1.0 / math.sqrt(D))
    yr.backward(g.float())
    assert (y.float() - yr).abs().max() <= 3e-2 and (x.grad.float() - xr.grad).abs().max() <= 3e-2 * xr.grad.abs().max()


@pytest.mark.parametrize("D", [64, 128])
def test_flash_many_sequences(native_lib, D):
    """More sequences than a warp has lanes, empty ones among them and at both ends."""
    from rl_b200.ops import functional as F
    from rl_b200.ops.lib import check_status

    lens = [0] + [(7 * i) % 5 * 37 + i % 3 for i in range(71)] + [0, 0]
    Hq, Hkv = 4, 2
    qkv, cu, D = _case(lens, Hq, Hkv, seed=5, D=D)
    x = qkv.clone().requires_grad_()
    y = F.attention_varlen(x, cu, max(lens), Hq, Hkv, D)
    g = torch.randn_like(y)
    y.backward(g)
    torch.cuda.synchronize()
    assert check_status() == 0
    xr = qkv.float().requires_grad_()
    yr = F._attention_ref(xr, cu, Hq, Hkv, D, 1.0 / math.sqrt(D))
    yr.backward(g.float())
    assert (y.float() - yr).abs().max() <= 3e-2 and (x.grad.float() - xr.grad).abs().max() <= 3e-2 * xr.grad.abs().max()


@pytest.mark.parametrize("D", [128, 64])
def test_flash_more_tiles_than_a_grid_dimension(native_lib, D):
    """65600 sequences of one token and two of 200, one of them last: more tiles than the second dimension of a grid can count. A token on its own
    gets its value, hands its gradient on to it (one bf16 rounding of a product with 1) and nothing to its query and key; the others as in
    test_flash_bwd_few_tiles."""
    from rl_b200.ops import functional as F
    from rl_b200.ops.lib import check_status

    n = 65600
    qkv, cu, D = _case([200] + [1] * n + [200], 1, 1, seed=D, D=D)
    x = qkv.clone().requires_grad_()
    y = F.attention_varlen(x, cu, 200, 1, 1, D)
    g = torch.randn_like(y)
    y.backward(g)
    torch.cuda.synchronize()
    assert check_status() == 0
    one = slice(200, 200 + n)
    assert torch.equal(y[one], qkv[one, 2 * D :]) and torch.equal(x.grad[one, 2 * D :], g[one]) and float(x.grad[one, : 2 * D].abs().max()) <= 1e-2
    for part in (slice(0, 200), slice(200 + n, 400 + n)):
        xr = qkv[part].float().requires_grad_()
        yr = F._attention_ref(xr, torch.tensor([0, 200], dtype=torch.int32, device="cuda"), 1, 1, D, 1.0 / math.sqrt(D))
        yr.backward(g[part].float())
        assert (y[part].float() - yr).abs().max() <= 3e-2 and (x.grad[part].float() - xr.grad).abs().max() <= 3e-2 * xr.grad.abs().max()


@pytest.mark.parametrize("D", [128, 64])
@pytest.mark.parametrize("n", [1, 16, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128])
@pytest.mark.parametrize("before", [0, 128, 256])
def test_flash_bwd_cut_tiles(native_lib, n, before, D):
    """Tiles of which only the first warps' rows, or the first half of the other side, belong to the sequence, alone and as the last of several. Bounds
    and repeats as in test_flash_bwd_few_tiles."""
    test_flash_bwd_few_tiles(native_lib, before + n, 4, 2, D)
