"""Mixture-of-experts compute: padded-by-expert token layout + grouped GEMMs (rl_b200/csrc/gemm_grouped.cu).

``grouped_expert_mlp(xs, counts, gate_up, down)`` runs the SwiGLU MLP of every local expert over its slice of ``xs``
(tokens sorted by expert, ``counts[e]`` rows each) with three launches in forward (two grouped GEMMs + SwiGLU) and no host
synchronisation: the per-expert segments are re-laid out with zero padding to multiples of 128 rows, so each 128-row tile
of the grouped GEMM belongs to one expert, and the tile -> expert table is computed on the device from ``counts``.
Weight gradients use the reduction form of the grouped GEMM and accumulate straight into the stacked gradient buffers.
``expert_layer`` is the whole layer on one rank, from tokens to tokens, with the rows planned, gathered and combined by kernels of its own.
On CPU (and for dtypes other than bf16) the per-expert loop of plain linears is used.
"""

from __future__ import annotations

import torch

from rl_b200.ops import functional as F
from rl_b200.ops import lib as _L
from rl_b200.ops.lib import I, L, P, call, ptr, register, stream_ptr, use_native

BF16 = torch.bfloat16
register("rlb_gemm_grouped_rows", [P, L, P, I, P, L, I, I, I, I, P, I, P, P])
register("rlb_gemm_grouped_reduce", [P, L, P, L, P, I, I, I, I, P, P, I, I, P, P])


class ExpertLayout:
    """Padded-by-expert row layout derived (on the device) from the per-expert row counts."""

    def __init__(self, counts: torch.Tensor, n_rows: int):
        E = counts.numel()
        dev = counts.device
        counts = counts.to(torch.int64)
        self.n_rows = n_rows
        self.num_experts = E
        self.mpad = -(-(n_rows + E * 127) // 128) * 128          # static upper bound: no host sync
        padded = (counts + 127) // 128 * 128
        ends = torch.cumsum(padded, 0)
        self.row0 = (ends - padded).to(torch.int32)
        self.rows = padded.to(torch.int32)
        start = torch.cumsum(counts, 0) - counts
        e_of_row = torch.repeat_interleave(torch.arange(E, device=dev), counts, output_size=n_rows)
        self.dest = (self.row0.long()[e_of_row] + torch.arange(n_rows, device=dev) - start[e_of_row])  # [n_rows] int64
        tile_start = torch.arange(self.mpad // 128, device=dev) * 128
        te = torch.searchsorted(ends, tile_start, right=True)
        self.tile_expert = torch.where(tile_start < ends[-1], te, torch.full_like(te, -1)).to(torch.int32)


class _GroupedLinear(torch.autograd.Function):
    """Y[Mpad, N] = X[Mpad, K] @ W[e(row)]^T with W stacked [E, N, K]."""

    @staticmethod
    def forward(ctx, x, w, lay: ExpertLayout):
        E, N, K = w.shape
        y = torch.zeros((lay.mpad, N), dtype=BF16, device=x.device)
        call("rlb_gemm_grouped_rows", ptr(x), x.stride(0), ptr(w), 0, ptr(y), y.stride(0), lay.mpad, N, K, E, ptr(lay.tile_expert), 0,
             ptr(_L.status_word(x.device)), stream_ptr())
        ctx.save_for_backward(x, w)
        ctx.lay = lay
        return y

    @staticmethod
    def backward(ctx, dy):
        x, w = ctx.saved_tensors
        lay = ctx.lay
        E, N, K = w.shape
        dy = dy if (dy.stride(-1) == 1 and dy.dtype == BF16) else dy.contiguous().to(BF16)
        dx = dw = None
        if ctx.needs_input_grad[0]:
            dx = torch.zeros((lay.mpad, K), dtype=BF16, device=dy.device)
            call("rlb_gemm_grouped_rows", ptr(dy), dy.stride(0), ptr(w), 1, ptr(dx), dx.stride(0), lay.mpad, K, N, E, ptr(lay.tile_expert),
                 0, ptr(_L.status_word(dy.device)), stream_ptr())
        if ctx.needs_input_grad[1]:
            main_grad, add = F.grad_output(w, dy.shape[0])
            target = main_grad if main_grad is not None else torch.zeros((E, N, K), dtype=torch.float32, device=dy.device)
            call("rlb_gemm_grouped_reduce", ptr(dy), dy.stride(0), ptr(x), x.stride(0), ptr(target), lay.mpad, N, K, E, ptr(lay.row0),
                 ptr(lay.rows), int(target.dtype == torch.float32), int(add), ptr(_L.status_word(dy.device)), stream_ptr())
            dw = None if main_grad is not None else target.to(w.dtype)
        return dx, dw, None


def grouped_linear(x_padded: torch.Tensor, w: torch.Tensor, lay: ExpertLayout) -> torch.Tensor:
    return _GroupedLinear.apply(x_padded, w, lay)


def grouped_expert_mlp(xs: torch.Tensor, counts: torch.Tensor, gate_up: torch.Tensor, down: torch.Tensor) -> torch.Tensor:
    """``xs`` [n, d] sorted by (local) expert, ``counts`` [E] rows per expert (device tensor), ``gate_up`` [E, 2f, d],
    ``down`` [E, d, f]. Returns the experts' outputs [n, d] in the order of ``xs``. Parameters that carry quantisation-aware
    training quantizers (``rl_b200/policy/qat.py``) have them applied to their weights and to the rows entering them."""
    n, d = xs.shape
    E = gate_up.shape[0]
    if n == 0:
        return xs.new_zeros((0, d))
    q_up, q_down = getattr(gate_up, "_rlb_qat", None), getattr(down, "_rlb_qat", None)
    if q_up is not None or q_down is not None:
        from rl_b200.policy.qat import QatState

        if not QatState.enabled:
            q_up = q_down = None
    if q_up is not None:
        xs, gate_up = q_up.q_input(xs), q_up.q_weight(gate_up)
    if q_down is not None:
        down = q_down.q_weight(down)
    native = use_native(xs) and xs.dtype == BF16 and d % 64 == 0 and down.shape[2] % 64 == 0
    if not native:
        outs, s = [], 0
        for e, c in enumerate(counts.tolist()):
            if c:
                xe = xs[s : s + c]
                a = F.swiglu(F.linear(xe, gate_up[e]))
                outs.append(F.linear(a if q_down is None else q_down.q_input(a), down[e]))
                s += c
        return torch.cat(outs, 0) if outs else xs.new_zeros((0, d))
    lay = ExpertLayout(counts, n)
    xp = torch.zeros((lay.mpad, d), dtype=xs.dtype, device=xs.device).index_copy(0, lay.dest, xs)
    h = grouped_linear(xp, gate_up, lay)
    a = F.swiglu(h)
    if q_down is not None:
        a = q_down.q_input(a)
    y = grouped_linear(a, down, lay)
    return y.index_select(0, lay.dest)


# ------------------------------------------------------------------------------------------- whole layer on one rank
register("rlb_moe_plan", [P, I, I, I, P, P, P, P, P, P, P])
register("rlb_moe_gather", [P, L, P, P, I, P, I, I, P])
register("rlb_moe_combine_rows", [P, P, P, P, L, P, L, I, I, P])
register("rlb_moe_combine_rows_bwd", [P, P, P, P, P, I, P, P, I, I, P])
LAYER_MAX_EXPERTS = 256


class TokenPlan:
    """Rows of the grouped GEMMs for the copies of ``idx`` [T, k] (int64 experts), made on the device: ``copy_row`` [T * k], ``row_copy``
    [mpad] (-1: padding), the experts' row ranges and the tile -> expert table."""

    def __init__(self, idx: torch.Tensor, num_experts: int):
        self.T, self.k = idx.shape
        n, dev = idx.numel(), idx.device
        self.num_experts = num_experts
        self.mpad = -(-(n + num_experts * 127) // 128) * 128          # static upper bound: no host sync
        blocks, E = -(-n // 1024), num_experts
        # one allocation: [scratch | copy_row | row_copy | row0 | rows | tile_expert]
        sizes = [blocks * E, n, self.mpad, E, E, self.mpad // 128]
        buf = torch.empty(sum(sizes), dtype=torch.int32, device=dev)
        scratch, self.copy_row, self.row_copy, self.row0, self.rows, self.tile_expert = buf.split(sizes)
        idx = idx.contiguous()
        call("rlb_moe_plan", ptr(idx), n, E, self.mpad, ptr(scratch), ptr(self.copy_row), ptr(self.row_copy), ptr(self.row0), ptr(self.rows),
             ptr(self.tile_expert), stream_ptr())


def _grouped_rows(x, w, transposed: bool, plan) -> torch.Tensor:
    """Rows of ``x`` times their expert's weight (``transposed``: [E, K, N] as stored, for the input gradient)."""
    E, N, K = w.shape
    if transposed:
        N, K = K, N
    y = torch.empty((plan.mpad, N), dtype=BF16, device=x.device)      # rows of unused tiles stay unwritten and are never read
    call("rlb_gemm_grouped_rows", ptr(x), x.stride(0), ptr(w), int(transposed), ptr(y), y.stride(0), plan.mpad, N, K, E, ptr(plan.tile_expert), 0,
         ptr(_L.status_word(x.device)), stream_ptr())
    return y


def _grouped_wgrad(dy, x, w, plan):
    """Adds the stacked weight gradient into ``w.main_grad``, or returns it."""
    E, N, K = w.shape
    main_grad, add = F.grad_output(w, dy.shape[0])
    target = main_grad if main_grad is not None else torch.zeros((E, N, K), dtype=torch.float32, device=dy.device)
    call("rlb_gemm_grouped_reduce", ptr(dy), dy.stride(0), ptr(x), x.stride(0), ptr(target), plan.mpad, N, K, E, ptr(plan.row0), ptr(plan.rows),
         int(target.dtype == torch.float32), int(add), ptr(_L.status_word(dy.device)), stream_ptr())
    return None if main_grad is not None else target.to(w.dtype)


class _ExpertLayer(torch.autograd.Function):
    """residual + sum of a token's experts' SwiGLU units, weighted (rl_b200/csrc/moe_layer.cu around the grouped GEMMs)."""

    @staticmethod
    def forward(ctx, x, w, residual, gate_up, down, plan: TokenPlan):
        d, f, dev = x.shape[1], down.shape[2], x.device
        xp = torch.empty((plan.mpad, d), dtype=BF16, device=dev)
        call("rlb_moe_gather", ptr(x), x.stride(0), ptr(plan.row_copy), ptr(plan.tile_expert), plan.k, ptr(xp), plan.mpad, d, stream_ptr())
        h = _grouped_rows(xp, gate_up, False, plan)
        a = torch.empty((plan.mpad, f), dtype=BF16, device=dev)
        call("rlb_swiglu_fwd", ptr(h), ptr(a), plan.mpad, f, stream_ptr())
        y = _grouped_rows(a, down, False, plan)
        out = torch.empty((plan.T, d), dtype=BF16, device=dev)
        call("rlb_moe_combine_rows", ptr(y), ptr(plan.copy_row), ptr(w), ptr(residual), residual.stride(0) if residual is not None else 0, ptr(out), plan.T,
             plan.k, d, stream_ptr())
        ctx.save_for_backward(w, gate_up, down, xp, h, a, y)
        ctx.plan = plan
        return out

    @staticmethod
    def backward(ctx, dout):
        w, gate_up, down, xp, h, a, y = ctx.saved_tensors
        plan, (d, f), dev = ctx.plan, (xp.shape[1], a.shape[1]), xp.device
        g = dout.contiguous()
        g = g if g.data_ptr() % 16 == 0 else g.clone()
        dy, dw = torch.empty_like(y), torch.zeros_like(w)
        call("rlb_moe_combine_rows_bwd", ptr(g), ptr(y), ptr(plan.row_copy), ptr(plan.tile_expert), ptr(w), plan.k, ptr(dy), ptr(dw), plan.mpad, d, stream_ptr())
        d_down = _grouped_wgrad(dy, a, down, plan) if ctx.needs_input_grad[4] else None
        dx = d_gate_up = None
        if ctx.needs_input_grad[0] or ctx.needs_input_grad[3]:
            da, dh = _grouped_rows(dy, down, True, plan), torch.empty_like(h)
            call("rlb_swiglu_bwd", ptr(da), ptr(h), ptr(dh), plan.mpad, f, stream_ptr())
            if ctx.needs_input_grad[3]:
                d_gate_up = _grouped_wgrad(dh, xp, gate_up, plan)
            if ctx.needs_input_grad[0]:
                dxp, dx = _grouped_rows(dh, gate_up, True, plan), torch.empty((plan.T, d), dtype=BF16, device=dev)
                call("rlb_moe_combine_rows", ptr(dxp), ptr(plan.copy_row), None, None, 0, ptr(dx), plan.T, plan.k, d, stream_ptr())
        return dx, dw, (dout if ctx.needs_input_grad[2] else None), d_gate_up, d_down, None


def expert_layer_takes(x: torch.Tensor, gate_up: torch.Tensor, down: torch.Tensor) -> bool:
    """Whether :func:`expert_layer` covers these rows and weights (bf16 on the GPU, widths in whole 64-column blocks, no quantizers)."""
    return (use_native(x) and x.dtype == BF16 and gate_up.dtype == BF16 and x.shape[0] > 0 and x.shape[1] % 64 == 0 and down.shape[2] % 64 == 0
            and gate_up.shape[0] <= LAYER_MAX_EXPERTS and getattr(gate_up, "_rlb_qat", None) is None and getattr(down, "_rlb_qat", None) is None)


def expert_layer(x: torch.Tensor, idx: torch.Tensor, w: torch.Tensor, residual, gate_up: torch.Tensor, down: torch.Tensor) -> torch.Tensor:
    """(residual +) sum_j w[t, j] MLP_{idx[t, j]}(x[t]) for tokens ``x`` [T, d]; ``idx``, ``w`` [T, k]. The sum over a token's experts is fp32
    and in their order."""
    def rows(t):      # (contiguous() would leave rows that start at an odd place where they are)
        fits = t is None or (t.stride(1) == 1 and t.stride(0) % 8 == 0 and t.data_ptr() % 16 == 0 and t.dtype == BF16)
        return t if fits else t.to(BF16).clone(memory_format=torch.contiguous_format)

    return _ExpertLayer.apply(rows(x), w.float().contiguous(), rows(residual), gate_up, down, TokenPlan(idx, gate_up.shape[0]))


# ------------------------------------------------------------------------------------------- small-token path (decode)
register("rlb_moe_route_topk", [P, L, I, I, I, I, P, P, P])
register("rlb_moe_decode_plan", [P, I, I, I, I, I, I, P, P, P, P, P, P, P])
register("rlb_moe_skinny", [P, L, P, P, L, I, I, I, I, I, P, I, P, P])
register("rlb_moe_gather_rows", [P, L, P, P, P, I, I, P])
register("rlb_moe_combine", [P, P, P, P, P, I, I, I, P])

SMALL_MAX_COPIES = 16384   # token copies (tokens x top-k, all ranks) the one-CTA layout kernel handles
SMALL_WORKSPACES: dict = {}  # single-rank workspaces by (device, hidden, inter, experts, top-k)


def route_topk_ref(logits: torch.Tensor, k: int, renorm: bool):
    probs = torch.softmax(logits.float(), dim=-1)
    w, idx = torch.topk(probs, k, dim=-1)
    return (w / w.sum(-1, keepdim=True) if renorm else w), idx.to(torch.int32)


def route_topk(logits: torch.Tensor, k: int, renorm: bool, out_w=None, out_idx=None):
    """Soft-max over the router logits [T, E] (bf16), the k largest probabilities and their experts (one kernel)."""
    if not (use_native(logits) and logits.dtype == BF16 and logits.stride(-1) == 1):
        return route_topk_ref(logits, k, renorm)
    T, E = logits.shape
    w = out_w if out_w is not None else torch.empty((T, k), dtype=torch.float32, device=logits.device)
    idx = out_idx if out_idx is not None else torch.empty((T, k), dtype=torch.int32, device=logits.device)
    call("rlb_moe_route_topk", ptr(logits), logits.stride(0), T, E, k, int(renorm), ptr(w), ptr(idx), stream_ptr())
    return w, idx


class SmallTokenMoE:
    """Buffers and launchers of the few-token MoE layer (rl_b200/csrc/moe_decode.cu): gather the tokens of all expert-
    parallel ranks, route them identically everywhere, run the local experts' grouped MLP over the copies routed to them
    and reduce the partial sums to the tokens' owners. Seven to nine launches per layer, fixed shapes, no host visit: a decode
    step that contains it can be captured in a CUDA graph. One instance serves all layers of a model.

    With ``ep.world > 1`` every rank of the group must call :meth:`forward` with the same number of tokens (the generation
    engine pads its decode batches to a bucket the ranks agree on)."""

    def __init__(self, hidden: int, inter: int, num_experts: int, top_k: int, ep, max_tokens: int, device, wait_limit_s: float = 20.0):
        self.d, self.f, self.E, self.k = hidden, inter, num_experts, top_k
        self.ep = ep
        self.W = ep.world if ep is not None else 1
        self.rank = ep.rank if ep is not None else 0
        self.El = num_experts // self.W
        self.e_lo = self.rank * self.El
        self.maxT = int(max_tokens)
        self.device = device
        self.wait_limit_s = wait_limit_s
        n_all = self.W * self.maxT
        assert n_all * top_k <= SMALL_MAX_COPIES and hidden % 8 == 0 and self.El <= 256 and top_k <= 16
        self.max_mpad = max(self.mpad_for(self.maxT), -(-(n_all * top_k + self.El * 127) // 128) * 128)
        i32 = dict(dtype=torch.int32, device=device)
        self.w = torch.empty((n_all, top_k), dtype=torch.float32, device=device)
        self.src_tok = torch.empty(self.max_mpad, **i32)
        self.copy_row = torch.empty(n_all * top_k, **i32)
        self.tile_expert = torch.empty(self.max_mpad // 32, **i32)
        self.row0 = torch.empty(self.El, **i32)
        self.rows = torch.empty(self.El, **i32)
        self.xp = torch.empty((self.max_mpad, hidden), dtype=BF16, device=device)
        self.h = torch.empty((self.max_mpad, 2 * inter), dtype=BF16, device=device)
        self.y = torch.empty((self.max_mpad, hidden), dtype=BF16, device=device)
        self._sym = []
        if self.W > 1:
            import ctypes as C

            from rl_b200.parallel.symmetric import SymmetricBuffer

            lib = _L.lib()
            Pp, Ii, LL, D = C.c_void_p, C.c_int, C.c_longlong, C.c_double
            lib.rlb_p2p_gather_cols.argtypes = [Pp, Pp, Pp, Pp, LL, Ii, Ii, Ii, Ii, Pp, D, Pp, Pp, LL, Pp]
            lib.rlb_p2p_gather_cols.restype = C.c_int
            lib.rlb_moe_combine_reduce.argtypes = [Pp, Pp, Pp, Pp, Pp, Ii, Ii, Ii, Pp, Pp, Ii, Ii, Pp, D, Pp, Pp, LL, Pp]
            lib.rlb_moe_combine_reduce.restype = C.c_int
            self._lib = lib
            self.stage_x = SymmetricBuffer(2 * self.maxT * hidden * 2, ep.group)
            self.stage_y = SymmetricBuffer(2 * n_all * hidden * 4, ep.group)
            self.flags = SymmetricBuffer(256, ep.group)          # words 0..7: gather, words 32..39: reduce
            self._sym = [self.stage_x, self.stage_y, self.flags]
            self._flags_g = (C.c_void_p * self.W)(*self.flags.peer_ptrs)
            self._flags_r = (C.c_void_p * self.W)(*[p + 128 for p in self.flags.peer_ptrs])
            self.epochs = torch.zeros(2, dtype=torch.int32, device=device)
            self.scratch = torch.zeros(2, dtype=torch.int32, device=device)
            self.x_all = torch.empty((n_all, hidden), dtype=BF16, device=device)

    def tile_rows(self, T: int) -> int:
        """Rows of a tile. Few tokens per expert: 32 or 64, the columns of the weight-streaming products (twice the mean load, so that nearly every
        expert's weights are read once, also where the routing is uneven); above a mean of 32 the 128-row tiles of the grouped GEMM. Whole layer, 8 of
        128 experts a token, width 2048, 768 per expert, even routing, us in tiles of 32 / 64 / 128: a mean of 2 231 / 239 / 311, 8 265 / 273 / 360,
        16 285 / 296 / 379, 24 306 / 315 / 397, 32 346 / 328 / 416, 48 457 / 358 / 453, 64 565 / 438 / 492. One rank's layer has at most 256 tokens,
        so means above 16 need few experts or several ranks; there tiles of 64 would still be ahead with experts like these."""
        mean = self.W * T * self.k / self.E
        if mean > 32 or self.d % 64 or self.f % 64:      # (the weight-streaming products have whole 64-column blocks)
            return 128
        return 32 if mean <= 16 else 64

    def mpad_for(self, T: int) -> int:
        pad = self.tile_rows(T)
        return -(-(self.W * T * self.k + self.El * (pad - 1)) // pad) * pad

    def fits(self, T: int) -> bool:
        return 0 < T <= self.maxT

    def forward(self, x: torch.Tensor, residual, router: torch.Tensor, gate_up: torch.Tensor, down: torch.Tensor, renorm: bool):
        """x [T, d] bf16 -> (residual +) MoE(x) [T, d]; also returns the top-k experts of this rank's tokens."""
        T, d = x.shape
        W, k = self.W, self.k
        n_all = W * T
        st = stream_ptr()
        status = ptr(_L.status_word(x.device))
        x = x if x.stride(1) == 1 and x.stride(0) == d else x.contiguous()
        if W > 1:
            xa = self.x_all[:n_all]
            rc = self._lib.rlb_p2p_gather_cols(x.data_ptr(), self.stage_x.table, self._flags_g, xa.data_ptr(), n_all * d * 2, 1, T * d * 2,
                                               self.rank, W, self.epochs[0:1].data_ptr(), float(self.wait_limit_s),
                                               self.scratch[0:1].data_ptr(), status, self.maxT * d * 2, st)
            _L.Counters.launches += 1
            if rc:
                raise RuntimeError(f"rlb_p2p_gather_cols failed with code {rc}")
        else:
            xa = x
        logits = F.linear(xa, router)
        wts, idx = self.w[:n_all], torch.empty((n_all, k), dtype=torch.int32, device=x.device)      # (the experts outlive the call)
        call("rlb_moe_route_topk", ptr(logits), logits.stride(0), n_all, self.E, k, int(renorm), ptr(wts), ptr(idx), st)
        mpad, pad = self.mpad_for(T), self.tile_rows(T)
        call("rlb_moe_decode_plan", ptr(idx), n_all * k, k, self.e_lo, self.El, mpad, pad, ptr(self.src_tok), ptr(self.copy_row),
             ptr(self.tile_expert), ptr(self.row0), ptr(self.rows), status, st)
        xp, y = self.xp[:mpad], self.y[:mpad]
        call("rlb_moe_gather_rows", ptr(xa), xa.stride(0) * 2, ptr(self.src_tok), ptr(self.tile_expert) if pad == 128 else None, ptr(xp), mpad, d * 2, st)
        if pad < 128:
            a = self.h.view(-1)[: mpad * self.f].view(mpad, self.f)
            call("rlb_moe_skinny", ptr(xp), xp.stride(0), ptr(gate_up), ptr(a), a.stride(0), mpad, pad, self.f, d, self.El, ptr(self.tile_expert), 1, status, st)
            call("rlb_moe_skinny", ptr(a), a.stride(0), ptr(down), ptr(y), y.stride(0), mpad, pad, d, self.f, self.El, ptr(self.tile_expert), 0, status, st)
        else:
            h = self.h[:mpad]
            call("rlb_gemm_grouped_rows", ptr(xp), xp.stride(0), ptr(gate_up), 0, ptr(h), h.stride(0), mpad, 2 * self.f, d, self.El,
                 ptr(self.tile_expert), 0, status, st)
            a = F.swiglu(h)
            call("rlb_gemm_grouped_rows", ptr(a), a.stride(0), ptr(down), 0, ptr(y), y.stride(0), mpad, d, self.f, self.El,
                 ptr(self.tile_expert), 0, status, st)
        out = torch.empty((T, d), dtype=BF16, device=x.device)
        res = ptr(residual.contiguous()) if residual is not None else None
        if W > 1:
            rc = self._lib.rlb_moe_combine_reduce(y.data_ptr(), self.copy_row.data_ptr(), wts.data_ptr(), res, out.data_ptr(), T, k, d,
                                                  self.stage_y.table, self._flags_r, self.rank, W, self.epochs[1:2].data_ptr(),
                                                  float(self.wait_limit_s), self.scratch[1:2].data_ptr(), status, W * self.maxT * d * 4, st)
            _L.Counters.launches += 1
            if rc:
                raise RuntimeError(f"rlb_moe_combine_reduce failed with code {rc}")
            mine = idx[self.rank * T : (self.rank + 1) * T]
        else:
            call("rlb_moe_combine", ptr(y), ptr(self.copy_row), ptr(wts), res, ptr(out), T, k, d, st)
            mine = idx
        return out, mine

    def close(self) -> None:
        for b in self._sym:
            b.close()
        self._sym = []
