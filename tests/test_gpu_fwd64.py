"""Attention forward for head_dim 64 (four CTAs per SM, steps of 64 keys) at the edges of its tiles, against a 64-bit result."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _dense(q, k, v, scale, pos, k_off, causal):
    q, k, v = q.double(), k.double(), v.double()
    g = q.shape[2] // k.shape[2]
    s = torch.einsum("bqhd,bkhd->bhqk", q, k.repeat_interleave(g, 2)) * scale
    if causal:
        s = s.masked_fill(pos[:, None] < torch.arange(k_off, k_off + k.shape[1], device=q.device)[None], float("-inf"))
    lse = torch.logsumexp(s, -1)
    p = torch.exp(s - torch.where(lse.isinf(), 0.0, lse)[..., None])
    return torch.einsum("bhqk,bkhd->bqhd", p, v.repeat_interleave(g, 2)), lse


@pytest.mark.parametrize("Tk", [1, 63, 64, 65, 129, 320, 700])
@pytest.mark.parametrize("Tq", [1, 127, 129, 300])
@pytest.mark.parametrize("mode", ["causal", "full", "offset", "ring"])
def test_tile_edges(Tq, Tk, mode):
    from context_parallelism_b200 import _native as nv
    from context_parallelism_b200.ops import attention as A
    g = torch.Generator(device="cuda").manual_seed(1000 * Tq + Tk)
    # scores of a spread that moves the running maximum by more than 2^8 between steps: the accumulators are rescaled
    q, k, v = (torch.randn(2, T, H, 64, device="cuda", generator=g).mul(f).bfloat16() for T, H, f in ((Tq, 6, 4), (Tk, 2, 4), (Tk, 2, 1)))
    pos = torch.arange(Tq, device="cuda")
    k_off = Tq // 2 if mode == "offset" else 0
    if mode == "ring":
        pos = torch.cat([pos[:Tq // 2], pos[Tq // 2:] + Tk // 2])
    o, lse = A.flash_fwd(q, k, v, 0.125, mode != "full", pos.int() if mode == "ring" else None, k_off)
    want, wl = _dense(q, k, v, 0.125, pos, k_off, mode != "full")
    # P is rounded to bf16 (2^-9) before its product and the result after it; scores of size 100 leave 1e-5 in fp32
    assert float((o.double() - want).norm() / want.norm().clamp(min=1e-9)) < 5e-3
    seen = ~wl.isinf()
    assert bool((lse.isinf() == ~seen).all()) and float((lse.double() - wl)[seen].abs().max() if seen.any() else 0.0) < 5e-5
    assert not bool(o.transpose(1, 2)[~seen].any())
    nv.status_for(q.device).check("forward")


def _plan(B, Tq, Tk, Hq, Hkv, causal=True, q_pos=False):
    from context_parallelism_b200 import _native as nv
    return nv.lib().cpb_flash_fwd_plan(B, Tq, Tk, Hq, Hkv, 64, int(causal), int(q_pos))


@pytest.mark.parametrize("Tk", [1, 63, 64, 65, 129, 320, 700])
@pytest.mark.parametrize("Tq", [1, 129, 300])
@pytest.mark.parametrize("mode", ["causal", "full", "offset", "ring"])
def test_tile_edges_with_four_ctas_per_sm(Tq, Tk, mode):
    """The cases above with the smallest batch for which the rule takes the kernel, and the batch below it, which it leaves to two CTAs."""
    from context_parallelism_b200 import _native as nv
    from context_parallelism_b200.ops import attention as A
    causal, ring = mode != "full", mode == "ring"
    B = next(b for b in range(1, 5000) if _plan(b, Tq, Tk, 6, 2, causal, ring) == 2)
    assert _plan(B - 1, Tq, Tk, 6, 2, causal, ring) == 0
    g = torch.Generator(device="cuda").manual_seed(1000 * Tq + Tk)
    q, k, v = (torch.randn(B, T, H, 64, device="cuda", generator=g).mul_(f).bfloat16() for T, H, f in ((Tq, 6, 4), (Tk, 2, 4), (Tk, 2, 1)))
    pos = torch.arange(Tq, device="cuda")
    k_off = Tq // 2 if mode == "offset" else 0
    if ring:
        pos = torch.cat([pos[:Tq // 2], pos[Tq // 2:] + Tk // 2])
    args = (0.125, causal, pos.int() if ring else None, k_off)
    o, lse = A.flash_fwd(q, k, v, *args)
    err = ref = worst = 0.0
    for b in range(0, B, 64):                                        # the 64-bit result of some sequences at a time
        part = slice(b, b + 64)
        want, wl = _dense(q[part], k[part], v[part], 0.125, pos, k_off, causal)
        err, ref = err + float((o[part].double() - want).norm() ** 2), ref + float(want.norm() ** 2)
        seen = ~wl.isinf()
        assert bool((lse[part].isinf() == ~seen).all()) and not bool(o[part].transpose(1, 2)[~seen].any())
        worst = max(worst, float((lse[part].double() - wl)[seen].abs().max()) if seen.any() else 0.0)
    assert err ** 0.5 <= 5e-3 * max(ref ** 0.5, 1e-9) and worst < 5e-5           # as above
    o2, lse2 = A.flash_fwd(q[1:], k[1:], v[1:], *args)
    # both lie within 5e-3 of the 64-bit result
    assert float((o2.float() - o[1:].float()).norm()) <= 1e-2 * max(float(o[1:].float().norm()), 1e-9)
    assert float((lse2 - lse[1:]).nan_to_num(0, 0, 0).abs().max()) < 1e-4
    nv.status_for(q.device).check("forward")
