"""Attention backward with several CTAs per K/V tile against whole sweeps and a 64-bit result."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _dense(q, k, v, do, scale, pos, k_off, causal):
    q, k, v = (t.double().requires_grad_() for t in (q, k, v))
    g = q.shape[2] // k.shape[2]
    s = torch.einsum("bqhd,bkhd->bhqk", q, k.repeat_interleave(g, 2)) * scale
    if causal:
        hidden = pos[:, None] < torch.arange(k_off, k_off + k.shape[1], device=q.device)[None]
        p = torch.softmax(s.masked_fill(hidden, -1e300), -1) * ~hidden              # a row that sees nothing is zero
    else:
        p = torch.softmax(s, -1)
    o = torch.einsum("bhqk,bkhd->bqhd", p, v.repeat_interleave(g, 2))
    return torch.autograd.grad(o, (q, k, v), do.double())


def _force(monkeypatch, AB, chunk):
    monkeypatch.setattr(AB, "bwd_chunk", lambda *a: chunk)
    monkeypatch.setattr(AB, "_bwd_plan", AB._bwd_plan.__wrapped__)      # without its cache


def _rel(a, b):
    return float((a.double() - b).norm() / b.norm().clamp(min=1e-30))


# chunk: fewer than, as many as and more than the pairs of a tile; odd, so that parts begin inside a head
@pytest.mark.parametrize("chunk", [0, 1, 3, 5, 1000])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Tq,Tk,Hq,Hkv,causal,k_off,ring", [
    (2, 300, 300, 6, 2, True, 0, False), (1, 128, 640, 4, 1, False, 0, False), (1, 257, 129, 2, 2, True, 0, False),
    (1, 256, 512, 4, 2, True, 100, True), (1, 200, 300, 3, 1, True, 180, False)])
def test_parts(monkeypatch, B, Tq, Tk, Hq, Hkv, causal, k_off, ring, D, chunk):
    from context_parallelism_b200 import _native as nv
    from context_parallelism_b200.ops import attention as A, attention_bwd as AB
    g = torch.Generator(device="cuda").manual_seed(Tq + Tk + D)
    q, k, v, do = (torch.randn(B, T, H, D, device="cuda", generator=g).bfloat16() for T, H in ((Tq, Hq), (Tk, Hkv), (Tk, Hkv), (Tq, Hq)))
    pos = torch.cat([torch.arange(128), torch.arange(384, 384 + Tq - 128)]).cuda() if ring else torch.arange(Tq, device="cuda")
    qp = pos.int() if ring else None
    scale = D ** -0.5
    o, lse = A.flash_fwd(q, k, v, scale, causal, qp, k_off)
    _force(monkeypatch, AB, chunk)
    got = AB.flash_bwd_cuda(q, k, v, o, lse, do, scale, causal, qp, k_off)
    for a, b in zip(got, _dense(q, k, v, do, scale, pos, k_off, causal)):
        # P and dS are rounded to bf16 (2^-9 each) before products whose terms partly cancel: 2.5e-3 is what whole sweeps have
        assert a.shape == b.shape and a.is_contiguous() and _rel(a, b) < 5e-3
    assert all(torch.equal(a, b) for a, b in zip(got[1:], AB.flash_bwd_cuda(q, k, v, o, lse, do, scale, causal, qp, k_off)[1:]))      # dK, dV repeat
    if not ring and Tq == Tk and k_off == 0:
        packed = torch.cat([q, k, v], 2)
        for x in (packed, packed.transpose(0, 1).contiguous().transpose(0, 1)):      # dense, and a layout that takes three gradients
            p = AB.flash_bwd_packed(x, Hq, Hkv, o, lse, do, scale, causal)
            for a, b in zip((p[:, :, :Hq], p[:, :, Hq:Hq + Hkv], p[:, :, Hq + Hkv:]), got):
                assert _rel(a, b.double()) < 2e-3                     # order of the fp32 sums, then one rounding
    nv.status_for(q.device).check("parts")


@pytest.mark.parametrize("B,T,Hq,Hkv,D", [(2, 1000, 6, 2, 64), (1, 2049, 4, 1, 64), (1, 1100, 4, 1, 128), (1, 4000, 8, 2, 128)])
def test_rule_and_no_loss_of_precision(monkeypatch, B, T, Hq, Hkv, D):
    from context_parallelism_b200.ops import attention as A, attention_bwd as AB
    assert AB.bwd_chunk(B, T, T, Hq, Hkv, D, True, 0, True) > 0
    assert AB.bwd_chunk(1, 32768, 32768, 32, 8, D, True, 0, True) == 0
    g = torch.Generator(device="cuda").manual_seed(T)
    q, k, v, do = (torch.randn(B, T, H, D, device="cuda", generator=g).bfloat16() for H in (Hq, Hkv, Hkv, Hq))
    o, lse = A.flash_fwd(q, k, v, D ** -0.5)
    args = (q, k, v, o, lse, do, D ** -0.5)
    got = AB.flash_bwd_cuda(*args)
    _force(monkeypatch, AB, 0)
    whole = AB.flash_bwd_cuda(*args)
    for a, w, b in zip(got, whole, _dense(q, k, v, do, D ** -0.5, torch.arange(T, device="cuda"), 0, True)):
        assert _rel(a, b) < 1.02 * _rel(w, b) + 1e-5
