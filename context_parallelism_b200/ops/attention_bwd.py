"""Host wrapper of the tcgen05 flash-attention backward (``csrc/kernels/attention_bwd.cu``)."""
from __future__ import annotations

import functools
import os
from typing import Optional

import torch

from .. import _native as nv
from .attention import _ok_layout, _strides

_INT_MAX = 2 ** 31 - 1
# CPB_BWD_GENERAL=1 routes head_dim 64 through the general kernel as well (comparison / fallback)
_USE_GENERAL_D64 = os.environ.get("CPB_BWD_GENERAL", "0") == "1"


def padded_q_pos(Tq: int, device, q_pos: Optional[torch.Tensor]) -> torch.Tensor:
    tq_pad = (Tq + 127) // 128 * 128
    out = torch.full((tq_pad,), _INT_MAX, dtype=torch.int32, device=device)
    if q_pos is None:
        out[:Tq] = torch.arange(Tq, dtype=torch.int32, device=device)
    else:
        out[:Tq] = q_pos.to(torch.int32)
    return out


def bwd_chunk(B: int, Tq: int, Tk: int, Hq: int, Hkv: int, D: int, causal: bool, k_off: int, local: bool) -> int:
    """Pairs of (query head, query tile) per CTA of the backward kernel, 0 for whole sweeps (the library's rule)."""
    return nv.lib().cpb_flash_bwd_chunk(B, Tq, Tk, Hq, Hkv, D, int(causal), k_off, int(local))


def flash_bwd_prep(o: torch.Tensor, do: torch.Tensor, lse: torch.Tensor, dq: Optional[torch.Tensor] = None,
                   q_pos: Optional[torch.Tensor] = None, qpos_pad: Optional[torch.Tensor] = None):
    """``delta = rowsum(dO∘O)`` and ``lse·log2(e)`` padded to a multiple of 128 rows.  The same launch clears the fp32
    accumulator ``dq`` (any contiguous tensor of a multiple of four values) and fills ``qpos_pad`` as :func:`padded_q_pos` does, when they are given."""
    B, Tq, Hq, D = o.shape
    tq_pad = (Tq + 127) // 128 * 128
    delta = torch.empty((B, Hq, tq_pad), dtype=torch.float32, device=o.device)
    lse2 = torch.empty_like(delta)
    nv.call("flash_bwd_prep", nv.ptr(o), nv.ptr(do), nv.ptr(lse), nv.ptr(delta), nv.ptr(lse2), nv.ptr(dq),
            0 if dq is None else dq.numel(), nv.ptr(q_pos), nv.ptr(qpos_pad), nv.i(B), nv.i(Tq), nv.i(Hq), nv.i(D), nv.i(tq_pad), nv.stream_ptr(o.device))
    return delta, lse2


def flash_bwd_delta(o: torch.Tensor, do: torch.Tensor) -> torch.Tensor:
    """Only ``delta = rowsum(dO∘O)`` ``[B,Hq,Tq_pad]`` (computed where the tokens live)."""
    B, Tq, Hq, D = o.shape
    tq_pad = (Tq + 127) // 128 * 128
    delta = torch.empty((B, Hq, tq_pad), dtype=torch.float32, device=o.device)
    nv.call("flash_bwd_prep", nv.ptr(o), nv.ptr(do), nv.ptr(None), nv.ptr(delta), nv.ptr(None), nv.ptr(None), 0, nv.ptr(None), nv.ptr(None),
            nv.i(B), nv.i(Tq), nv.i(Hq), nv.i(D), nv.i(tq_pad), nv.stream_ptr(o.device))
    return delta


def flash_bwd_lse2(lse: torch.Tensor, D: int) -> torch.Tensor:
    """Only ``lse·log2(e)`` padded ``[B,Hq,Tq_pad]``."""
    B, Hq, Tq = lse.shape
    tq_pad = (Tq + 127) // 128 * 128
    lse2 = torch.empty((B, Hq, tq_pad), dtype=torch.float32, device=lse.device)
    nv.call("flash_bwd_prep", nv.ptr(None), nv.ptr(None), nv.ptr(lse), nv.ptr(None), nv.ptr(lse2), nv.ptr(None), 0, nv.ptr(None), nv.ptr(None),
            nv.i(B), nv.i(Tq), nv.i(Hq), nv.i(D), nv.i(tq_pad), nv.stream_ptr(lse.device))
    return lse2


def flash_bwd_core(q, k, v, do, lse2, delta, qpos_pad, scale, causal, k_off, dq_f32, dk, dv, dkv_accumulate,
                   route=None, dkv_st: int = 0):
    """One launch of the backward kernel: ``dq_f32`` (fp32) is accumulated with atomics; ``dk``/``dv`` are
    written as bf16, or accumulated in fp32 when ``dkv_accumulate``.  ``route = (route_k, route_v, rows, tl)``
    (int64 device tables of per-chunk owner addresses) makes the epilogue add each dK/dV tile into its owner's
    fp32 accumulator over NVLink instead.  ``dkv_st`` is the distance between two tokens of ``dk`` / ``dv`` in elements
    (default: dense)."""
    B, Tq, Hq, D = q.shape
    Tk, Hkv = k.shape[1], k.shape[2]
    st = nv.status_for(q.device)
    qs, ks = _strides(q), _strides(k)
    assert v.stride() == k.stride()
    if D == 64 and not _USE_GENERAL_D64:
        nv.call("flash_bwd64", nv.ptr(q), nv.ptr(k), nv.ptr(v), nv.ptr(do), nv.ptr(lse2), nv.ptr(delta), nv.ptr(dq_f32),
                nv.ptr(dk), nv.ptr(dv), nv.i(B), nv.i(Tq), nv.i(Tk), nv.i(Hq), nv.i(Hkv), nv.i(lse2.shape[-1]),
                nv.l(qs[0]), nv.l(qs[1]), nv.l(qs[2]), nv.l(ks[0]), nv.l(ks[1]), nv.l(ks[2]),
                nv.f(scale), nv.i(causal), nv.i(k_off), nv.ptr(qpos_pad), nv.i(2 if route is not None else int(dkv_accumulate)), nv.l(dkv_st or Hkv * D),
                nv.ptr(route[0] if route else None), nv.ptr(route[1] if route else None),
                nv.i(route[2] if route else 0), nv.i(route[3] if route else 0), 0, 0, st.ptr(), nv.stream_ptr(q.device))
        return
    if D == 128:
        nv.call("flash_bwd128", nv.ptr(q), nv.ptr(k), nv.ptr(v), nv.ptr(do), nv.ptr(lse2), nv.ptr(delta), nv.ptr(dq_f32),
                nv.ptr(dk), nv.ptr(dv), nv.i(B), nv.i(Tq), nv.i(Tk), nv.i(Hq), nv.i(Hkv), nv.i(lse2.shape[-1]),
                nv.l(qs[0]), nv.l(qs[1]), nv.l(qs[2]), nv.l(ks[0]), nv.l(ks[1]), nv.l(ks[2]),
                nv.f(scale), nv.i(causal), nv.i(k_off), nv.ptr(qpos_pad), nv.i(2 if route is not None else int(dkv_accumulate)), nv.l(dkv_st or Hkv * D),
                nv.ptr(route[0] if route else None), nv.ptr(route[1] if route else None),
                nv.i(route[2] if route else 0), nv.i(route[3] if route else 0), 0, 0, st.ptr(), nv.stream_ptr(q.device))
        return
    assert dkv_st in (0, Hkv * D), "the general kernel writes dense dK/dV"
    nv.call("flash_bwd", nv.ptr(q), nv.ptr(k), nv.ptr(v), nv.ptr(do), nv.ptr(lse2), nv.ptr(delta), nv.ptr(dq_f32),
            nv.ptr(dk), nv.ptr(dv), nv.i(B), nv.i(Tq), nv.i(Tk), nv.i(Hq), nv.i(Hkv), nv.i(D), nv.i(lse2.shape[-1]),
            nv.l(qs[0]), nv.l(qs[1]), nv.l(qs[2]), nv.l(ks[0]), nv.l(ks[1]), nv.l(ks[2]),
            nv.f(scale), nv.i(causal), nv.i(k_off), nv.ptr(qpos_pad), nv.i(2 if route is not None else int(dkv_accumulate)),
            nv.ptr(route[0] if route else None), nv.ptr(route[1] if route else None),
            nv.i(route[2] if route else 0), nv.i(route[3] if route else 0), st.ptr(), nv.stream_ptr(q.device))


def cast_to_bf16(x_f32: torch.Tensor, scale: float = 1.0) -> torch.Tensor:
    out = torch.empty(x_f32.shape, dtype=torch.bfloat16, device=x_f32.device)
    nv.call("cast_f32_bf16", nv.ptr(x_f32), nv.ptr(out), nv.l(x_f32.numel()), nv.f(scale), nv.stream_ptr(x_f32.device))
    return out


def _launch_ready(q, k, v):
    if not _ok_layout(q):
        q = q.contiguous()
    if not _ok_layout(k):
        k = k.contiguous()
    if not _ok_layout(v) or v.stride() != k.stride():
        v = v.contiguous()
        if v.stride() != k.stride():
            k = k.contiguous()
    return q, k, v


def _aligned(t: torch.Tensor) -> torch.Tensor:
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


@functools.lru_cache(maxsize=4096)
def _bwd_plan(B: int, Tq: int, Tk: int, Hq: int, Hkv: int, D: int, causal: bool, k_off: int, local: bool):
    """``(pairs per CTA, floats of workspace)`` of a whole gradient."""
    chunk, tq_pad = bwd_chunk(B, Tq, Tk, Hq, Hkv, D, causal, k_off, local), (Tq + 127) // 128 * 128
    parts = -(-(Hq // Hkv * tq_pad // 128) // chunk) if chunk else 0
    return chunk, B * D * (Tq * Hq + 2 * parts * Tk * Hkv) + (2 * B * Hq + 1) * tq_pad


def _bwd_whole(q: int, k: int, v: int, o, do, lse, dq: int, dk: int, dv: int, dims, strides, dq_st: int, dkv_st: int, scale: float, causal: bool,
               k_off: int, q_pos) -> None:
    """Preparation, kernel and cast behind one call of the library; ``q`` .. ``dv`` are addresses, ``strides`` those of q and of k/v."""
    chunk, floats = _bwd_plan(*dims, bool(causal), k_off, q_pos is None)
    dev = o.device
    ws = torch.empty(floats, dtype=torch.float32, device=dev)
    nv.LAUNCHES[0] += 2                                              # three kernels
    nv.call("flash_attn_bwd", q, k, v, o.data_ptr(), do.data_ptr(), lse.data_ptr(), ws.data_ptr(), dq, dk, dv, *dims, *strides, dq_st, dkv_st,
            scale, int(causal), k_off, nv.ptr(q_pos), chunk, nv.status_for(dev).ptr(), nv.stream_ptr(dev))


def flash_bwd_cuda(q, k, v, o, lse, do, scale, causal=True, q_pos=None, k_off=0,
                   dq=None, dk=None, dv=None, dkv_accumulate=False):
    B, Tq, Hq, D = q.shape
    Tk, Hkv = k.shape[1], k.shape[2]
    q, k, v = _launch_ready(q, k, v)
    do, o = _aligned(do), _aligned(o)
    pos32 = None if q_pos is None else q_pos.to(torch.int32).contiguous()
    # a launch timer (nv.profile_start) wants the launches one by one
    if dq is None and not dkv_accumulate and nv._PROFILE is None and not (D == 64 and _USE_GENERAL_D64):
        dq = torch.empty((B, Tq, Hq, D), dtype=torch.bfloat16, device=q.device)
        dk = torch.empty((B, Tk, Hkv, D), dtype=torch.bfloat16, device=q.device)
        dv = torch.empty_like(dk)
        _bwd_whole(q.data_ptr(), k.data_ptr(), v.data_ptr(), o, do, lse, dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), (B, Tq, Tk, Hq, Hkv, D),
                   (*_strides(q), *_strides(k)), Hq * D, Hkv * D, scale, causal, k_off, pos32)
        return dq, dk, dv
    dq_f32 = torch.empty((B, Tq, Hq, D), dtype=torch.float32, device=q.device) if dq is None else dq
    qpos_pad = torch.empty((Tq + 127) // 128 * 128, dtype=torch.int32, device=q.device)
    delta, lse2 = flash_bwd_prep(o, do, lse, dq_f32 if dq is None else None, pos32, qpos_pad)
    if dkv_accumulate:
        assert dk is not None and dv is not None and dk.dtype == torch.float32
    else:
        dk = torch.empty((B, Tk, Hkv, D), dtype=torch.bfloat16, device=q.device)
        dv = torch.empty_like(dk)
    flash_bwd_core(q, k, v, do, lse2, delta, qpos_pad, scale, causal, k_off, dq_f32, dk, dv, dkv_accumulate)
    if dq is None:
        return cast_to_bf16(dq_f32), dk, dv
    return dq_f32, dk, dv


def flash_bwd_packed(qkv: torch.Tensor, Hq: int, Hkv: int, o, lse, do, scale: float, causal: bool = True) -> torch.Tensor:
    """Gradient of packed projections ``qkv`` (``[B,T,Hq+2·Hkv,D]`` or ``[B,T,(Hq+2·Hkv)·D]``: query heads, then key heads, then value
    heads), every part written where it belongs: three separate gradients cost autograd a zero-filled full-size tensor and a copy
    each, and two full-size additions."""
    B, T, H = qkv.shape[0], qkv.shape[1], Hq + 2 * Hkv
    W = qkv.shape[2] * (qkv.shape[3] if qkv.dim() == 4 else 1)
    D = W // H
    if nv._PROFILE is None and not (D == 64 and _USE_GENERAL_D64) and qkv.is_contiguous() and qkv.data_ptr() % 16 == 0:
        dqkv = torch.empty_like(qkv)
        x, g, k_at, v_at = qkv.data_ptr(), dqkv.data_ptr(), 2 * Hq * D, 2 * (Hq + Hkv) * D
        _bwd_whole(x, x + k_at, x + v_at, _aligned(o), _aligned(do), lse, g, g + k_at, g + v_at, (B, T, T, Hq, Hkv, D),
                   (D, W, T * W, D, W, T * W), W, W, scale, causal, 0, None)
        return dqkv
    x, heads = qkv.view(B, T, H, D), (B, T, Hq, D)
    grads = flash_bwd_cuda(x[:, :, :Hq], x[:, :, Hq:Hq + Hkv], x[:, :, Hq + Hkv:], o.reshape(heads), lse, do.reshape(heads), scale, causal)
    return torch.cat(grads, 2).view(qkv.shape)
