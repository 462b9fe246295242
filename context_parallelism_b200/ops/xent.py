"""Fused language-model head + cross-entropy that never materialises ``[tokens, vocab]``.

``linear_cross_entropy(x, w, targets)`` returns the *sum* of token NLLs (fp32).  On CUDA the rows are processed in chunks: the lm_head
GEMM leaves (max, sum of exponentials) of each row and column tile (``gemm_head``), ``xent_rows`` turns them into losses and the rows'
gradient coefficients, and for gradients the bf16 dlogits come from a second GEMM with the same epilogue or, for wide hidden states,
from logits that the first one stored (``xent_dlogits``); a dX chunk GEMM and the accumulation of dW follow.  All of it happens inside
the forward call (the gradient of a sum-of-NLL loss with respect to the logits does not depend on anything downstream except one
scalar, which is applied in ``backward``).  The reference materialises the full logits tensor (Scripts/Blutrain/bluscriptCP.cpp:452-459),
which at T = 128 K and a 128 K vocabulary would be 64 GB.
"""
from __future__ import annotations

from typing import Optional

import torch
import torch.nn.functional as F

from .. import _native as nv
from .gemm import _rowmajor2d, gemm

CHUNK_ROWS = 4096
# Up to this width of the hidden states the gradient pass computes the logits a second time instead of reading them back.  Whole call, 4096
# rows, us, stored and computed again: width 384, 50304 columns 793 and 654; 768 954 and 911; 1024 1150 and 1161 (128256 columns 3027 and
# 3080); 1280 1582 and 1751; 2048, 128256 columns 5724 and 6338.  Before either, with a cross entropy of its own that kept each row in
# a cluster's shared memory: 384 873, 768 1037, 1280 1900, 2048 5900; losses alone 383, 425, 599, 1984, now 174, 218, 472, 1650.
RECOMPUTE_WIDTH = 1024


def xent_chunk(logits: torch.Tensor, targets: torch.Tensor, loss_sum: torch.Tensor, grad_scale: float,
               want_grad: bool = True, row_loss: torch.Tensor = None, n_valid: int = 0):
    """Cross entropy of fp32 logits that the caller has in memory: loss and bf16 dlogits in one launch.  The head does not store them whole
    and does not come by here."""
    rows, Vc = logits.shape
    V = n_valid or Vc
    dlog = torch.empty((rows, Vc), dtype=torch.bfloat16, device=logits.device) if want_grad else None
    st = nv.status_for(logits.device)
    nv.call("xent", nv.ptr(logits), nv.ptr(targets), nv.ptr(dlog), nv.ptr(loss_sum), nv.ptr(row_loss), nv.i(rows), nv.i(V), nv.i(Vc),
            nv.l(logits.stride(0)), nv.l(dlog.stride(0) if dlog is not None else 0), nv.f(grad_scale), st.ptr(),
            nv.stream_ptr(logits.device))
    return dlog


HEAD_TILE = 256          # columns per tile of the head's GEMM


def _head_operands(x: torch.Tensor, w: torch.Tensor, targets: torch.Tensor):
    """``x`` and ``w`` as the head's GEMM takes them, and 64-bit targets: the launchers get addresses and know neither types nor widths."""
    assert x.dtype == torch.bfloat16 and w.dtype == torch.bfloat16, f"the head computes in bf16 (got {x.dtype} and {w.dtype})"
    assert w.device == x.device and targets.device == x.device, f"operands on {x.device}, {w.device} and {targets.device}"
    x2, w2, tg = _rowmajor2d(x), _rowmajor2d(w), targets.reshape(-1).contiguous().long()
    assert x2.shape[1] == w2.shape[1], f"hidden states of width {x2.shape[1]}, weights of width {w2.shape[1]}"
    assert tg.numel() >= x2.shape[0], f"{tg.numel()} targets for {x2.shape[0]} rows"
    return x2, w2, tg


def _head_rows(xc: torch.Tensor, w: torch.Tensor, tg: torch.Tensor, n_valid: int, grad_scale: float, loss_sum: Optional[torch.Tensor],
               row_loss: Optional[torch.Tensor], want_coef: bool, logits: Optional[torch.Tensor] = None) -> Optional[torch.Tensor]:
    """Loss of the rows ``xc`` (``loss_sum`` += , ``row_loss`` =); returns the rows' gradient coefficients.  ``logits`` (fp32) are stored only
    when given."""
    rows, V = xc.shape[0], w.shape[0]
    tiles = (V + HEAD_TILE - 1) // HEAD_TILE
    stats = torch.empty((tiles, rows, 2), dtype=torch.float32, device=xc.device)
    tlogit = torch.empty(rows, dtype=torch.float32, device=xc.device)
    coef = torch.empty((rows, 2), dtype=torch.float32, device=xc.device) if want_coef else None
    st, stream = nv.status_for(xc.device).ptr(), nv.stream_ptr(xc.device)
    nv.call("gemm_head", xc.data_ptr(), w.data_ptr(), nv.ptr(logits), tg.data_ptr(), stats.data_ptr(), tlogit.data_ptr(), 0, rows, V, xc.shape[1],
            xc.stride(0), w.stride(0), 0 if logits is None else logits.stride(0), n_valid, 0, grad_scale, st, stream)
    nv.call("xent_rows", stats.data_ptr(), tlogit.data_ptr(), tg.data_ptr(), nv.ptr(coef), nv.ptr(row_loss), nv.ptr(loss_sum), rows, tiles,
            n_valid, grad_scale, st, stream)
    return coef


def _head_dlogits(xc: torch.Tensor, w: torch.Tensor, tg: torch.Tensor, coef: torch.Tensor, n_valid: int, grad_scale: float,
                  logits: Optional[torch.Tensor] = None) -> torch.Tensor:
    """bf16 gradient of the logits, which are computed again unless they were stored."""
    dlog = torch.empty((xc.shape[0], w.shape[0]), dtype=torch.bfloat16, device=xc.device)
    if logits is not None:
        nv.call("xent_dlogits", logits.data_ptr(), tg.data_ptr(), coef.data_ptr(), dlog.data_ptr(), xc.shape[0], n_valid, w.shape[0],
                logits.stride(0), dlog.stride(0), grad_scale, nv.stream_ptr(xc.device))
        return dlog
    nv.call("gemm_head", xc.data_ptr(), w.data_ptr(), dlog.data_ptr(), tg.data_ptr(), 0, 0, coef.data_ptr(), xc.shape[0], w.shape[0], xc.shape[1],
            xc.stride(0), w.stride(0), dlog.stride(0), n_valid, 1, grad_scale, nv.status_for(xc.device).ptr(), nv.stream_ptr(xc.device))
    return dlog


class _LinearCEFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w, targets, grad_scale, n_valid):
        x2, wm, tg = _head_operands(x, w, targets)
        N, d = x2.shape
        V = w.shape[0]
        loss_sum = torch.zeros(1, dtype=torch.float32, device=x.device)
        need_grad = x.requires_grad or w.requires_grad
        dx = torch.empty_like(x2) if need_grad else None
        mg = getattr(w, "main_grad", None)
        dw_own = None
        if need_grad and mg is None:
            dw_own = torch.zeros((V, d), dtype=torch.float32, device=x.device)
        stored = need_grad and d > RECOMPUTE_WIDTH
        logits = torch.empty((min(CHUNK_ROWS, N), V), dtype=torch.float32, device=x.device) if stored else None
        for r0 in range(0, N, CHUNK_ROWS):
            r1 = min(N, r0 + CHUNK_ROWS)
            xc, tc = x2[r0:r1], tg[r0:r1]
            lg = logits[: r1 - r0] if stored else None
            coef = _head_rows(xc, wm, tc, n_valid or V, grad_scale, loss_sum, None, need_grad, lg)
            if need_grad:
                dlog = _head_dlogits(xc, wm, tc, coef, n_valid or V, grad_scale, lg)
                gemm(dlog, wm, b_mn=True, out=dx[r0:r1])
                gemm(dlog, xc, a_mn=True, b_mn=True, out=(mg if mg is not None else dw_own).view(V, d), accumulate=True)
        if need_grad and mg is not None:
            hook = getattr(w, "_grad_ready", None)
            if hook is not None:
                ctx.hook, ctx.w = hook, w
        ctx.dx = dx
        ctx.dw_own = dw_own
        ctx.grad_scale = grad_scale
        ctx.xshape = x.shape
        ctx.wdtype = w.dtype
        return loss_sum.squeeze(0)

    @staticmethod
    def backward(ctx, g):
        # dX/dW were produced with `grad_scale`; the upstream scalar must match it (checked lazily on the
        # device would cost a sync, so the contract is enforced by the callers in this package).
        hook = getattr(ctx, "hook", None)
        if hook is not None:
            hook(ctx.w)
        dx = ctx.dx.view(ctx.xshape) if ctx.dx is not None else None
        dw = ctx.dw_own.to(ctx.wdtype) if ctx.dw_own is not None else None
        return dx, dw, None, None, None


def linear_cross_entropy(x: torch.Tensor, w: torch.Tensor, targets: torch.Tensor, grad_scale: float = 1.0,
                         n_valid: int = 0) -> torch.Tensor:
    """Sum over tokens of ``-log softmax(x·wᵀ)[target]`` (targets < 0 are ignored).

    ``grad_scale`` is the scalar the caller will pass to ``backward`` for this loss (for a mean over
    ``n`` tokens and ``a`` accumulation steps: ``1/(n·a)``); on CUDA the gradients are produced during
    the forward with that factor folded in.  ``w`` may carry zero padding rows beyond the real vocabulary
    ``n_valid`` (kept so the GEMM shapes are multiples of 64); they never enter the softmax."""
    if x.is_cuda:
        return _LinearCEFn.apply(x, w, targets, grad_scale, n_valid)
    logits = F.linear(x.float(), w.float())
    if n_valid:
        logits = logits[..., :n_valid]
    return F.cross_entropy(logits.view(-1, logits.shape[-1]), targets.reshape(-1), ignore_index=-100, reduction="sum")


def per_token_nll(x: torch.Tensor, w: torch.Tensor, targets: torch.Tensor, n_valid: int = 0) -> torch.Tensor:
    """Forward-only per-token NLL ``[tokens]`` (per-position perplexity evaluation)."""
    if not x.is_cuda:
        logits = F.linear(x.reshape(-1, x.shape[-1]).float(), w.float())
        if n_valid:
            logits = logits[:, :n_valid]
        return F.cross_entropy(logits, targets.reshape(-1).long(), reduction="none")
    x2, wm, tg = _head_operands(x, w, targets)
    N, V = x2.shape[0], w.shape[0]
    out = torch.empty(N, dtype=torch.float32, device=x.device)
    for r0 in range(0, N, CHUNK_ROWS):
        r1 = min(N, r0 + CHUNK_ROWS)
        _head_rows(x2[r0:r1], wm, tg[r0:r1], n_valid or V, 1.0, None, out[r0:r1], False)
    return out


def logits_last(x_last: torch.Tensor, w: torch.Tensor) -> torch.Tensor:
    """fp32 logits for a few rows (generation)."""
    if not x_last.is_cuda:
        return F.linear(x_last.float(), w.float())
    return gemm(x_last.reshape(-1, x_last.shape[-1]), w, out_dtype=torch.float32)
