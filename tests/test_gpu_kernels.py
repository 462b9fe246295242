"""Numerics of each sm_100a kernel against a plain PyTorch fp32 reference of the same op."""
import math

import pytest
import torch

from util import assert_close

pytestmark = pytest.mark.gpu


def dev():
    return torch.device("cuda", 0)


def check_status():
    from context_parallelism_b200 import _native as nv
    torch.cuda.synchronize()
    nv.status_for(dev()).check()


@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (256, 512, 256), (1000, 384, 520), (4096, 2048, 2048), (72, 128, 64)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
def test_gemm_majors(M, N, K, a_mn, b_mn):
    from context_parallelism_b200.ops.gemm import gemm
    torch.manual_seed(0)
    A = torch.randn(M, K, device=dev()).bfloat16()
    B = torch.randn(N, K, device=dev()).bfloat16()
    want = A.float() @ B.float().t()
    a = A.t().contiguous() if a_mn else A
    b = B.t().contiguous() if b_mn else B
    got = gemm(a, b, a_mn=a_mn, b_mn=b_mn)
    check_status()
    assert_close(got.float(), want, cos=0.9999, rel=2e-2, name=f"gemm {M}x{N}x{K} a_mn={a_mn} b_mn={b_mn}")


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
def test_gemm_pair_banded_order(a_mn, b_mn):
    """A B operand above 64 MB switches the CTA-pair kernel to its banded tile order (8 pair-rows per band, a ragged last
    band here: 11 pair-rows); every output tile must still be produced exactly once."""
    from context_parallelism_b200.ops.gemm import gemm
    torch.manual_seed(3)
    M, N, K = 2816 - 8, 8192, 4160
    A = torch.randn(M, K, device=dev()).bfloat16()
    B = (torch.randn(N, K, device=dev()) * 0.1).bfloat16()
    want = A.float() @ B.float().t()
    a = A.t().contiguous() if a_mn else A
    b = B.t().contiguous() if b_mn else B
    got = gemm(a, b, a_mn=a_mn, b_mn=b_mn)
    check_status()
    assert_close(got.float(), want, cos=0.9999, rel=2e-2, name=f"banded gemm a_mn={a_mn} b_mn={b_mn}")


def test_gemm_epilogues():
    from context_parallelism_b200.ops import gemm as G
    torch.manual_seed(1)
    M, N, K = 512, 768, 384
    A = torch.randn(M, K, device=dev()).bfloat16()
    B = (torch.randn(N, K, device=dev()) * 0.05).bfloat16()
    bias = torch.randn(N, device=dev())
    ref = A.float() @ B.float().t()
    got = G.gemm(A, B, out_dtype=torch.float32, bias=bias)
    assert_close(got, ref + bias, cos=0.99999, rel=1e-3, name="f32+bias")
    acc = torch.ones(M, N, device=dev())
    G.gemm(A, B, out=acc, accumulate=True)
    assert_close(acc, ref + 1, cos=0.99999, rel=1e-3, name="f32 accumulate")
    pre = torch.empty(M, N, device=dev(), dtype=torch.bfloat16)
    act = G.gemm(A, B, bias=bias, epi=G.EPI_BF16_GELU, aux=pre)
    assert_close(pre.float(), ref + bias, cos=0.9999, rel=2e-2, name="gelu pre")
    assert_close(act.float(), torch.nn.functional.gelu(ref + bias, approximate="tanh"), cos=0.9999, rel=2e-2, name="gelu")
    Fh = N // 2
    gu = torch.empty(M, N, device=dev(), dtype=torch.bfloat16)
    sw = G.gemm(A, B, epi=G.EPI_BF16_SWIGLU, aux=gu)
    assert sw.shape == (M, Fh)
    assert_close(gu.float(), ref, cos=0.9999, rel=2e-2, name="swiglu pre")
    assert_close(sw.float(), torch.nn.functional.silu(ref[:, :Fh]) * ref[:, Fh:], cos=0.9999, rel=3e-2, name="swiglu")
    check_status()


# Edges of the tiles (256 x 128 / 256 rows, 64 of K), row counts below one CTA of a pair, and shapes whose weight gradient is
# split along K.  bf16 outputs: one rounding (2^-9) on top of fp32 sums.  fp32: two summation orders of K products of
# unit normals differ by about sqrt(K) * 2^-24 * sqrt(K), relative to the result's sqrt(K): 5e-6 at K = 8192.
@pytest.mark.parametrize("M,N,K", [(8, 264, 64), (136, 768, 776), (129, 8, 72), (257, 120, 64), (384, 384, 8192), (640, 392, 4104), (520, 1288, 136)])
def test_gemm_tile_edges_every_epilogue(M, N, K):
    from context_parallelism_b200.ops import gemm as G
    torch.manual_seed(17)
    A = torch.randn(M, K, device=dev()).bfloat16()
    B = torch.randn(N, K, device=dev()).bfloat16()
    bias = torch.randn(N, device=dev())
    ref = (A.double() @ B.double().t()).float()
    rms = K ** 0.5
    got = G.gemm(A, B, bias=bias)
    assert_close(got.float(), ref + bias, cos=0.99999, rel=2 ** -8, name="bf16 + bias")
    assert float((G.gemm(A, B, out_dtype=torch.float32, bias=bias) - ref - bias).abs().max()) < 1e-4 * rms
    pre = torch.empty(M, N, device=dev(), dtype=torch.bfloat16)
    act = G.gemm(A, B, bias=bias, epi=G.EPI_BF16_GELU, aux=pre)
    assert_close(pre.float(), ref + bias, cos=0.99999, rel=2 ** -8, name="gelu pre")
    want = torch.nn.functional.gelu((ref + bias).double(), approximate="tanh").float()
    assert_close(act.float(), want, cos=0.99999, rel=2 ** -8, name="gelu")
    assert torch.equal(G.gemm(A, B, bias=bias, epi=G.EPI_BF16_GELU), act)          # without the pre-activation
    if N % 16 == 0:
        F = N // 2
        gu = torch.empty(M, N, device=dev(), dtype=torch.bfloat16)
        sw = G.gemm(A, B, epi=G.EPI_BF16_SWIGLU, aux=gu)
        assert_close(gu.float(), ref, cos=0.99999, rel=2 ** -8, name="swiglu pre")
        want = torch.nn.functional.silu(ref[:, :F].double()).float() * ref[:, F:]
        assert_close(sw.float(), want, cos=0.99999, rel=2 ** -8, name="swiglu")
        assert torch.equal(G.gemm(A, B, epi=G.EPI_BF16_SWIGLU), sw)
    if M % 8 == 0:
        acc = torch.randn(M, N, device=dev())
        want = acc + ref
        G.gemm(A.t().contiguous(), B.t().contiguous(), a_mn=True, b_mn=True, out=acc, accumulate=True)
        assert float((acc - want).abs().max()) < 1e-4 * rms
    check_status()


@pytest.mark.parametrize("M,N,K", [(384, 384, 8192), (768, 768, 4096), (2048, 1024, 64)])      # twelve splits along K, four, none
def test_gemm_accumulate_adds_the_bias_once(M, N, K):
    from context_parallelism_b200.ops import gemm as G
    torch.manual_seed(18)
    A, B = torch.randn(M, K, device=dev()).bfloat16(), torch.randn(N, K, device=dev()).bfloat16()
    bias, acc = 100 * torch.randn(N, device=dev()), torch.randn(M, N, device=dev())
    want = acc.double() + A.double() @ B.double().t() + bias.double()
    G.gemm(A, B, out=acc, accumulate=True, bias=bias)
    check_status()
    # K products of unit normals in fp32: about sqrt(K) * 2^-24 * sqrt(K); two more roundings of values up to 500
    assert float((acc.double() - want).abs().max()) < 1e-6 * K + 2e-4


@pytest.mark.parametrize("M,N,K", [(384, 384, 8192), (1152, 384, 4096), (640, 392, 4104)])
def test_gemm_accumulate_repeats_bit_for_bit(M, N, K):
    """Weight gradients whose K range is split are added in a fixed order."""
    from context_parallelism_b200.ops import gemm as G
    torch.manual_seed(19)
    A, B = torch.randn(K, M, device=dev()).bfloat16(), torch.randn(K, N, device=dev()).bfloat16()
    start, runs = torch.randn(M, N, device=dev()), []
    for _ in range(20):
        acc = start.clone()
        G.gemm(A, B, a_mn=True, b_mn=True, out=acc, accumulate=True)
        runs.append(acc)
    check_status()
    assert all(torch.equal(r, runs[0]) for r in runs)


def test_gemm_activation_epilogues_over_the_range():
    """SwiGLU and GELU of single values from -80 to 80: one column of A times a row of ones gives every value exactly.  The bound
    is one rounding to bf16 (half a step of 8 significant bits, 2^-8) and a hundred fp32 ones (the exponential of 80); GELU is taken as 0.5 x (1 + tanh) in fp32, so its negative side
    is good to a few 2^-24 of x only."""
    from context_parallelism_b200.ops import gemm as G
    x = torch.linspace(-80, 80, 2048, device=dev()).bfloat16()
    A = torch.zeros(2048, 64, device=dev()).bfloat16()
    A[:, 0], A[:, 1] = x, 1.0
    W = torch.zeros(32, 64, device=dev()).bfloat16()
    W[:16, 0], W[16:, 1] = 1.0, 1.0                                    # gate = x, up = 1
    xd = x.double()
    sw = G.gemm(A, W, epi=G.EPI_BF16_SWIGLU)[:, 3].double()
    want = xd * torch.sigmoid(xd)
    assert bool(((sw - want).abs() <= want.abs() * (2.0 ** -8 + 2.0 ** -16)).all())
    ge = G.gemm(A, W[:16], epi=G.EPI_BF16_GELU)[:, 3].double()
    want = torch.nn.functional.gelu(xd, approximate="tanh")
    assert bool(((ge - want).abs() <= want.abs() * (2.0 ** -8 + 2.0 ** -16) + xd.abs() * 2.0 ** -21).all())
    check_status()


@pytest.mark.parametrize("M,N,K", [(136, 272, 72), (384, 384, 8192), (520, 1296, 136)])
def test_gemm_writes_into_wider_buffers(M, N, K):
    """C and the pre-activation as columns of wider buffers, every epilogue and a split accumulation: what dense outputs give, and
    nothing beside them."""
    from context_parallelism_b200.ops import gemm as G
    torch.manual_seed(20)
    A, B = torch.randn(M, K, device=dev()).bfloat16(), torch.randn(N, K, device=dev()).bfloat16()
    at, bt = A.t().contiguous(), B.t().contiguous()

    def wide(cols, dtype):
        buf = torch.full((M + 2, cols + 24), 7.0, device=dev(), dtype=dtype)
        return buf, buf[1:M + 1, 16:16 + cols]

    def untouched(buf, view, cols):
        view.fill_(7.0)
        return bool((buf == 7.0).all())
    bf, f32 = torch.bfloat16, torch.float32
    for kw, cols, dtype, aux in ((dict(), N, bf, 0), (dict(epi=G.EPI_F32), N, f32, 0), (dict(epi=G.EPI_BF16_GELU), N, bf, N),
                                 (dict(epi=G.EPI_BF16_SWIGLU), N // 2, bf, N), (dict(accumulate=True, a_mn=True, b_mn=True), N, f32, 0)):
        a, b = (at, bt) if "a_mn" in kw else (A, B)
        dense = torch.full((M, cols), 7.0, device=dev(), dtype=dtype)
        dense_aux = torch.empty(M, aux, device=dev(), dtype=bf) if aux else None
        buf, out = wide(cols, dtype)
        abuf, aout = wide(aux, bf) if aux else (None, None)
        G.gemm(a, b, out=dense, aux=dense_aux, **kw)
        G.gemm(a, b, out=out, aux=aout, **kw)
        check_status()
        assert torch.equal(out, dense) and untouched(buf, out, cols), kw
        if aux:
            assert torch.equal(aout, dense_aux) and untouched(abuf, aout, aux), kw


def test_linear_autograd():
    from context_parallelism_b200.ops.gemm import linear, linear_swiglu, linear_gelu
    torch.manual_seed(2)
    x = torch.randn(4, 96, 256, device=dev()).bfloat16().requires_grad_()
    w = (torch.randn(512, 256, device=dev()) * 0.05).bfloat16().requires_grad_()
    b = torch.randn(512, device=dev(), requires_grad=True)
    for fn, rf in ((lambda: linear(x, w, b), lambda X, W, Bb: torch.nn.functional.linear(X, W, Bb)),
                   (lambda: linear_gelu(x, w, b), lambda X, W, Bb: torch.nn.functional.gelu(torch.nn.functional.linear(X, W, Bb), approximate="tanh")),
                   (lambda: linear_swiglu(x, w), lambda X, W, Bb: torch.nn.functional.silu(torch.nn.functional.linear(X, W)[..., :256]) * torch.nn.functional.linear(X, W)[..., 256:])):
        x.grad = w.grad = b.grad = None
        y = fn()
        dy = torch.randn_like(y)
        y.backward(dy)
        X, W, Bb = x.detach().float().requires_grad_(), w.detach().float().requires_grad_(), b.detach().clone().requires_grad_()
        Y = rf(X, W, Bb)
        Y.backward(dy.float())
        assert_close(y.float(), Y, cos=0.9999, name="fwd")
        assert_close(x.grad.float(), X.grad, cos=0.999, name="dx")
        assert_close(w.grad.float(), W.grad, cos=0.999, name="dw")
        if Bb.grad is not None and b.grad is not None:
            assert_close(b.grad.float(), Bb.grad, cos=0.999, name="db")
    check_status()


@pytest.mark.parametrize("layer", [0, 1])
@pytest.mark.parametrize("d", [384, 768, 2048, 4096])
@pytest.mark.parametrize("with_res", [False, True])
def test_norm(layer, d, with_res):
    from context_parallelism_b200.ops import elementwise as E
    torch.manual_seed(3)
    rows = 300
    x = torch.randn(rows, d, device=dev()).bfloat16().requires_grad_()
    r = torch.randn(rows, d, device=dev()).bfloat16().requires_grad_() if with_res else None
    w = (1 + 0.1 * torch.randn(d, device=dev())).requires_grad_()
    b = (0.1 * torch.randn(d, device=dev())).requires_grad_() if layer else None
    y, xn = (E.layernorm(x, w, b, 1e-5, r) if layer else E.rmsnorm(x, w, 1e-5, r))
    dy, dxn = torch.randn_like(y), torch.randn_like(y)
    (y.float() * dy.float()).sum().backward() if False else torch.autograd.backward([y, xn], [dy, dxn])
    X = x.detach().float().requires_grad_()
    R = r.detach().float().requires_grad_() if with_res else None
    W = w.detach().clone().requires_grad_()
    Bb = b.detach().clone().requires_grad_() if layer else None
    XN = (X + R).bfloat16().float() if with_res else X
    if with_res:
        XN = X + R
    if layer:
        Y = torch.nn.functional.layer_norm(XN, (d,), W, Bb, 1e-5)
    else:
        Y = XN * torch.rsqrt(XN.pow(2).mean(-1, keepdim=True) + 1e-5) * W
    torch.autograd.backward([Y, XN], [dy.float(), dxn.float()])
    assert_close(y.float(), Y, cos=0.9999, rel=3e-2, name="y")
    assert_close(x.grad.float(), X.grad, cos=0.999, name="dx")
    if with_res:
        assert_close(r.grad.float(), R.grad, cos=0.999, name="dres")
    assert_close(w.grad, W.grad, cos=0.999, name="dw")
    if layer:
        assert_close(b.grad, Bb.grad, cos=0.999, name="db")


@pytest.mark.parametrize("D", [64, 128])
def test_qk_norm_rope(D):
    from context_parallelism_b200.ops import elementwise as E, reference as R
    torch.manual_seed(4)
    B, T, Hq, Hkv = 2, 96, 4, 2
    qkv = torch.randn(B, T, (Hq + 2 * Hkv) * D, device=dev()).bfloat16().requires_grad_()
    gq = (1 + 0.1 * torch.randn(D, device=dev())).requires_grad_()
    gk = (1 + 0.1 * torch.randn(D, device=dev())).requires_grad_()
    cache = R.build_rope_cache(512, D, 10000.0).to(dev())
    pos = torch.randint(0, 512, (T,), device=dev())
    out = E.qk_norm_rope(qkv, gq, gk, cache, pos, Hq, Hkv, D, 1e-6)
    dout = torch.randn_like(out)
    out.backward(dout)
    X = qkv.detach().float().cpu().requires_grad_()
    GQ, GK = gq.detach().cpu().requires_grad_(), gk.detach().cpu().requires_grad_()
    want = E.qk_norm_rope(X, GQ, GK, cache.cpu(), pos.cpu(), Hq, Hkv, D, 1e-6)
    want.backward(dout.float().cpu())
    assert_close(out.float().cpu(), want, cos=0.9999, rel=3e-2, name="fwd")
    assert_close(qkv.grad.float().cpu(), X.grad, cos=0.999, name="dqkv")
    assert_close(gq.grad.cpu(), GQ.grad, cos=0.999, name="dgq")
    assert_close(gk.grad.cpu(), GK.grad, cos=0.999, name="dgk")
    check_status()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Tq,Tk,Hq,Hkv,causal", [
    (1, 128, 128, 1, 1, False), (1, 128, 128, 1, 1, True), (2, 384, 384, 4, 2, True),
    (1, 200, 328, 2, 1, False), (1, 1024, 1024, 2, 2, True)])
def test_flash_fwd(D, B, Tq, Tk, Hq, Hkv, causal):
    from context_parallelism_b200.ops import attention as A, reference as R
    torch.manual_seed(5)
    q = torch.randn(B, Tq, Hq, D, device=dev()).bfloat16()
    k = torch.randn(B, Tk, Hkv, D, device=dev()).bfloat16()
    v = torch.randn(B, Tk, Hkv, D, device=dev()).bfloat16()
    scale = 1 / math.sqrt(D)
    out, lse = A.flash_fwd(q, k, v, scale, causal)
    check_status()
    want, wlse = R.attention_dense(q.float(), k.float(), v.float(), scale, causal=causal)
    assert_close(out.float(), want, cos=0.9995, rel=3e-2, name="out")
    assert_close(lse, wlse, cos=0.99999, rel=1e-3, name="lse")


def test_flash_fwd_positions_packed():
    """Global-position masking with a HeadTail query shard against a position-ordered K/V, consumed as
    strided views of a packed QKV buffer."""
    from context_parallelism_b200.ops import attention as A, reference as R
    from context_parallelism_b200.parallel.shard import local_positions
    torch.manual_seed(6)
    B, T, Hq, Hkv, D, N, r = 1, 1024, 4, 2, 64, 4, 1
    qkv = torch.randn(B, T, (Hq + 2 * Hkv), D, device=dev()).bfloat16()
    qfull, k, v = qkv[:, :, :Hq], qkv[:, :, Hq:Hq + Hkv], qkv[:, :, Hq + Hkv:]
    pos = local_positions(T, N, r, True).to(dev())
    q = qfull[:, pos].contiguous()
    out, lse = A.flash_fwd(q, k, v, 0.125, True, q_pos=pos.int())
    check_status()
    want, wlse = R.attention_dense(q.float(), k.float(), v.float(), 0.125, q_pos=pos, causal=True)
    assert_close(out.float(), want, cos=0.9995, rel=3e-2, name="out")
    assert_close(lse, wlse, cos=0.99999, rel=1e-3, name="lse")


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Tq,Tk,Hq,Hkv,causal", [
    (1, 128, 128, 1, 1, False), (1, 128, 128, 1, 1, True), (2, 384, 384, 4, 2, True),
    (1, 200, 328, 2, 1, False), (1, 1024, 1024, 4, 1, True)])
def test_flash_bwd(D, B, Tq, Tk, Hq, Hkv, causal):
    from context_parallelism_b200.ops import attention as A, reference as R
    torch.manual_seed(7)
    q = torch.randn(B, Tq, Hq, D, device=dev()).bfloat16()
    k = torch.randn(B, Tk, Hkv, D, device=dev()).bfloat16()
    v = torch.randn(B, Tk, Hkv, D, device=dev()).bfloat16()
    do = torch.randn(B, Tq, Hq, D, device=dev()).bfloat16()
    scale = 1 / math.sqrt(D)
    out, lse = A.flash_fwd(q, k, v, scale, causal)
    dq, dk, dv = A.flash_bwd(q, k, v, out, lse, do, scale, causal)
    check_status()
    want, wlse = R.attention_dense(q.float(), k.float(), v.float(), scale, causal=causal)
    wdq, wdk, wdv = R.attention_dense_bwd(q.float(), k.float(), v.float(), want, wlse, do.float(), scale, causal=causal)
    assert_close(dv.float(), wdv, cos=0.998, rel=5e-2, name="dv")
    assert_close(dk.float(), wdk, cos=0.998, rel=5e-2, name="dk")
    assert_close(dq.float(), wdq, cos=0.998, rel=5e-2, name="dq")


# Both head widths: one query tile, ragged ends on both sides, several tiles of several grouped heads (both stages of every ring
# in use), the zig-zag shard of a ring rank, a key block at an offset, rows that see no key.  Same bars as test_flash_bwd.
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Tq,Tk,Hq,Hkv,ring,k_off,accumulate", [
    (1, 1, 1, 1, 1, 1, 0, False), (2, 129, 127, 2, 1, 1, 0, True), (1, 640, 896, 4, 2, 1, 0, False), (1, 256, 1024, 6, 2, 4, 0, True),
    (2, 384, 200, 2, 2, 1, 100, False), (1, 130, 300, 3, 1, 1, 64, True)])
def test_flash_bwd_shapes_and_modes(D, B, Tq, Tk, Hq, Hkv, ring, k_off, accumulate):
    from context_parallelism_b200.ops import attention as A, reference as R
    from context_parallelism_b200.parallel.shard import local_positions
    torch.manual_seed(21)
    q = torch.randn(B, Tq, Hq, D, device=dev()).bfloat16()
    k, v = (torch.randn(B, Tk, Hkv, D, device=dev()).bfloat16() for _ in range(2))
    do = torch.randn(B, Tq, Hq, D, device=dev()).bfloat16()
    pos = local_positions(Tq * ring, ring, 1, True).to(dev()) if ring > 1 else torch.arange(Tq, device=dev())
    kpos = torch.arange(k_off, k_off + Tk, device=dev())
    scale = D ** -0.5
    out, lse = A.flash_fwd(q, k, v, scale, True, pos.int(), k_off)
    extra = {}
    if accumulate:
        extra = dict(dk=torch.ones(B, Tk, Hkv, D, device=dev()), dv=torch.ones(B, Tk, Hkv, D, device=dev()), dkv_accumulate=True)
    dq, dk, dv = A.flash_bwd(q, k, v, out, lse, do, scale, True, pos.int(), k_off, **extra)
    check_status()
    want, wlse = R.attention_dense(q.float(), k.float(), v.float(), scale, q_pos=pos, k_pos=kpos, causal=True)
    wdq, wdk, wdv = R.attention_dense_bwd(q.float(), k.float(), v.float(), want, wlse, do.float(), scale, q_pos=pos, k_pos=kpos, causal=True)
    off = 1.0 if accumulate else 0.0
    for got, ref, name in ((dv.float() - off, wdv, "dv"), (dk.float() - off, wdk, "dk"), (dq.float(), wdq, "dq")):
        assert torch.isfinite(got).all()
        if float(ref.abs().max()) > 1e-4:
            assert_close(got, ref, cos=0.998, rel=5e-2, name=name)
        else:
            # one key: P = 1 and dP = Delta up to two fp32 sums of D products, at most D * 2^-23 * 4 D = 8e-3 apart (values up to 2
            # on average at most); times a key or query (up to 5) and the scale (at most 1/8)
            assert float(got.abs().max()) < 5e-3, name


@pytest.mark.parametrize("B,Tq,Tk,Hq,Hkv,causal", [(1, 512, 512, 4, 1, True), (2, 300, 712, 2, 2, False), (1, 2048, 2048, 8, 2, True)])
def test_flash_bwd_d64_kernels_agree(B, Tq, Tk, Hq, Hkv, causal, monkeypatch):
    """The head_dim-64 kernel (transposed, in two query halves) against the general kernel on the same inputs,
    including the fp32-accumulating dK/dV mode; query positions of a zig-zag shard when causal."""
    from context_parallelism_b200.ops import attention as A, attention_bwd as AB
    from context_parallelism_b200.parallel.shard import local_positions
    torch.manual_seed(11)
    D = 64
    q = torch.randn(B, Tq, Hq, D, device=dev()).bfloat16()
    k = torch.randn(B, Tk, Hkv, D, device=dev()).bfloat16()
    v = torch.randn(B, Tk, Hkv, D, device=dev()).bfloat16()
    do = torch.randn(B, Tq, Hq, D, device=dev()).bfloat16()
    scale = 1 / math.sqrt(D)
    q_pos = None
    if causal and Tq == 512:
        q_pos = local_positions(4 * Tq, 4, 1, True).to(dev()).int()       # rank 1 of 4: chunks 1 and 6
        k = torch.randn(B, 4 * Tq, Hkv, D, device=dev()).bfloat16()
        v = torch.randn_like(k)
    out, lse = A.flash_fwd(q, k, v, scale, causal, q_pos=q_pos)
    got = {}
    for general in (True, False):
        monkeypatch.setattr(AB, "_USE_GENERAL_D64", general)
        got[general] = A.flash_bwd(q, k, v, out, lse, do, scale, causal, q_pos=q_pos)
        check_status()
    for a, b_, n in zip(got[True], got[False], ("dq", "dk", "dv")):
        assert torch.isfinite(b_.float()).all()
        assert_close(b_.float(), a.float(), cos=0.9995, rel=3e-2, name=n)


def test_flash_autograd_positions():
    from context_parallelism_b200.ops import attention as A
    from context_parallelism_b200.parallel.shard import local_positions
    torch.manual_seed(8)
    B, T, Hq, Hkv, D, N, r = 1, 1024, 4, 2, 64, 4, 2
    pos = local_positions(T, N, r, True).to(dev())
    q = torch.randn(B, T // N, Hq, D, device=dev()).bfloat16().requires_grad_()
    k = torch.randn(B, T, Hkv, D, device=dev()).bfloat16().requires_grad_()
    v = torch.randn(B, T, Hkv, D, device=dev()).bfloat16().requires_grad_()
    out, _ = A.flash_attention(q, k, v, None, True, pos.int())
    do = torch.randn_like(out)
    out.backward(do)
    check_status()
    Q, K, V = (t.detach().float().cpu().requires_grad_() for t in (q, k, v))
    want, _ = A.flash_attention(Q, K, V, None, True, pos.cpu())
    want.backward(do.float().cpu())
    assert_close(out.float().cpu(), want, cos=0.9995, name="out")
    for a, b_, n in ((q, Q, "dq"), (k, K, "dk"), (v, V, "dv")):
        assert_close(a.grad.float().cpu(), b_.grad, cos=0.998, name=n)


@pytest.mark.parametrize("D,Hq,Hkv", [(64, 4, 2), (128, 2, 1), (32, 4, 4)])
def test_attention_fp32_accurate_variant(D, Hq, Hkv):
    """ATTN_FP32 kernels: fp32 arithmetic on bf16 inputs reproduces the dense oracle far more tightly than the tensor-core
    path (forward cos > 0.99999 and 1e-3 relative, gradients cos > 0.9999: the reference's fp32 bars)."""
    from context_parallelism_b200.ops import attention as A
    from context_parallelism_b200.ops import reference as ref
    torch.manual_seed(3)
    B, T = 2, 200
    q, k, v, do = (torch.randn(B, T, h, D, device=dev()).bfloat16() for h in (Hq, Hkv, Hkv, Hq))
    scale = D ** -0.5
    qpos = torch.arange(T, device=dev()) + 7
    A.FP32_ACCURATE = True
    try:
        qi, ki, vi = (t.clone().requires_grad_() for t in (q, k, v))
        o, lse = A.flash_attention(qi, ki, vi, scale, True, qpos, 5)
        o.backward(do)
    finally:
        A.FP32_ACCURATE = False
    kp = torch.arange(5, 5 + T, device=dev())
    o_ref, lse_ref = ref.attention_dense(q.float(), k.float(), v.float(), scale, qpos, kp, True)
    g_ref = ref.attention_dense_bwd(q.float(), k.float(), v.float(), o_ref, lse_ref, do.float(), scale, qpos, kp, True)
    check_status()
    assert_close(o.float(), o_ref, cos=0.99999, rel=1e-2, name="fp32 attn out")       # the bf16 rounding of the output remains
    assert_close(lse, lse_ref, cos=0.999999, rel=1e-4, name="fp32 attn lse")
    for got, want, nm in zip((qi.grad, ki.grad, vi.grad), g_ref, ("dq", "dk", "dv")):
        assert_close(got.float(), want, cos=0.9999, rel=2e-2, name="fp32 attn " + nm)


# packed projections: every layout the packed gradient is written in (one and several KV heads, an odd number of rows, one row)
@pytest.mark.parametrize("B,T,Hq,Hkv,D", [(2, 200, 6, 2, 64), (1, 1, 2, 1, 64), (1, 129, 4, 4, 128), (2, 384, 3, 1, 128)])
def test_packed_attention_matches_separate(B, T, Hq, Hkv, D):
    """The same kernels either way: the output is equal, gradients differ by the order of the dQ additions only."""
    from context_parallelism_b200.ops import attention as A
    torch.manual_seed(5)
    qkv = torch.randn(B, T, (Hq + 2 * Hkv) * D, device=dev()).bfloat16()
    do = torch.randn(B, T, Hq * D, device=dev()).bfloat16()
    a, b = qkv.clone().requires_grad_(), qkv.clone().requires_grad_()
    out = A.flash_attention_packed(a, Hq, Hkv, D, D ** -0.5)
    x = b.view(B, T, Hq + 2 * Hkv, D)
    want, _ = A.flash_attention(x[:, :, :Hq], x[:, :, Hq:Hq + Hkv], x[:, :, Hq + Hkv:], D ** -0.5)
    out.backward(do)
    want.backward(do.view(B, T, Hq, D))
    check_status()
    assert torch.equal(out, want.view(B, T, Hq * D))
    nq = Hq * D
    assert torch.equal(a.grad[..., nq:], b.grad[..., nq:])                      # dK, dV: one writer, fixed order
    assert_close(a.grad[..., :nq].float(), b.grad[..., :nq].float(), cos=0.99999, rel=4e-3, name="dq")


def test_packed_attention_output_can_be_changed_in_place():
    from context_parallelism_b200.ops import attention as A
    qkv = torch.randn(1, 128, 4 * 64, device=dev()).bfloat16().requires_grad_()
    out = A.flash_attention_packed(qkv, 2, 1, 64, 0.125)
    want = out.detach() + 1
    out += 1                                    # a view made inside the autograd function would refuse this
    assert torch.equal(out.detach(), want)


def test_packed_attention_takes_the_heads_as_a_dimension_of_their_own():
    from context_parallelism_b200.ops import attention as A
    torch.manual_seed(7)
    qkv, do = torch.randn(2, 130, 8 * 64, device=dev()).bfloat16(), torch.randn(2, 130, 4 * 64, device=dev()).bfloat16()
    a, b = qkv.clone().requires_grad_(), qkv.view(2, 130, 8, 64).clone().requires_grad_()
    outs = [A.flash_attention_packed(x, 4, 2, 64, 0.125) for x in (a, b)]
    [o.backward(do) for o in outs]
    check_status()
    assert torch.equal(*outs) and torch.equal(a.grad[..., 256:], b.grad.view(2, 130, 512)[..., 256:])
    assert_close(a.grad.float(), b.grad.view(2, 130, 512).float(), cos=0.99999, rel=4e-3, name="dqkv")


@pytest.mark.parametrize("B,T,H,D,with_pos", [(2, 130, 3, 64, True), (1, 128, 2, 128, False), (1, 1, 1, 64, False)])
def test_flash_bwd_prep_outputs(B, T, H, D, with_pos):
    from context_parallelism_b200.ops import attention_bwd as AB
    torch.manual_seed(6)
    o, do = (torch.randn(B, T, H, D, device=dev()).bfloat16() for _ in range(2))
    lse = torch.randn(B, H, T, device=dev())
    lse[0, 0, T // 2] = -math.inf
    dq = torch.full((B, T, H, D), 7.0, device=dev())
    pos = torch.arange(T, device=dev(), dtype=torch.int32) * 3 if with_pos else None
    pad = (T + 127) // 128 * 128
    qp = torch.zeros(pad, dtype=torch.int32, device=dev())
    delta, lse2 = AB.flash_bwd_prep(o, do, lse, dq, pos, qp)
    assert float(dq.abs().max()) == 0.0
    assert torch.equal(qp, AB.padded_q_pos(T, dev(), pos))
    want = (o.double() * do.double()).sum(-1).transpose(1, 2)
    # fp32 sum of D products of bf16 values: D rounding errors of 2^-24 of the sum of magnitudes
    bound = (o.double() * do.double()).abs().sum(-1).transpose(1, 2) * D * 2.0 ** -24
    assert bool(((delta[..., :T].double() - want).abs() <= bound).all())
    assert bool((delta[..., T:] == 0).all()) and bool((lse2[..., T:] == math.inf).all())
    finite = lse != -math.inf
    assert torch.allclose(lse2[..., :T][finite], lse[finite] * 1.4426950408889634, rtol=1e-6)
    assert bool((lse2[..., :T][~finite] == math.inf).all())


# two query tiles per CTA (long key sequences, many CTAs): ragged query tiles, a zig-zag shard whose tiles see
# very different spans, an odd key count, and the wrapped sweep with readiness flags
@pytest.mark.parametrize("Tq,Tk,Hq,Hkv,causal,ring,flags", [
    (300, 8292, 120, 8, True, 0, False), (129, 8192, 240, 2, False, 0, False), (512, 8192, 120, 4, True, 16, False),
    (512, 8192, 120, 4, True, 16, True), (1000, 8199, 60, 1, True, 0, False)])
def test_flash_fwd_d128_pair_kernel(Tq, Tk, Hq, Hkv, causal, ring, flags):
    from context_parallelism_b200.ops import attention as A, reference as R
    from context_parallelism_b200.parallel.shard import local_positions
    torch.manual_seed(12)
    D = 128
    q = torch.randn(1, Tq, Hq, D, device=dev()).bfloat16()
    k, v = (torch.randn(1, Tk, Hkv, D, device=dev()).bfloat16() for _ in range(2))
    pos = local_positions(Tk, ring, 3, True).to(dev()) if ring else torch.arange(Tk - Tq, Tk, device=dev())
    extra = {}
    if flags:
        rows = Tk // (2 * ring)
        extra = dict(ready=torch.full((2 * ring,), 5, dtype=torch.int32, device=dev()), ready_epoch=5, block_rows=rows)
    out, lse = A.flash_fwd(q, k, v, D ** -0.5, causal, pos.int(), **extra)
    check_status()
    assert Hq * ((Tq + 255) // 256) * 2 >= 3 * torch.cuda.get_device_properties(0).multi_processor_count      # the rule's side
    want, wlse = R.attention_dense(q.float(), k.float(), v.float(), D ** -0.5, q_pos=pos, causal=causal)
    assert_close(out.float(), want, cos=0.9995, rel=3e-2, name="out")
    assert_close(lse, wlse, cos=0.99999, rel=1e-3, name="lse")


@pytest.mark.parametrize("poly,share", [(None, 2 / 8), ("0", 0.0), ("3", 3 / 8)])
def test_flash_fwd_d128_share_of_polynomial_exponentials(poly, share):
    """With all scores zero every exponential is 1, where the polynomial gives 1 - 7.24e-5: the LSE shows the share of columns that
    took it, for one query tile per CTA and for two, and CPB_FWD_POLY (read once per process) sets it for both."""
    import os
    import subprocess
    import sys
    code = ("import torch, math\nfrom context_parallelism_b200.ops import attention as A\n"
            "for Tq, Tk, H in ((256, 1024, 2), (512, 8192, 120)):\n"
            "    q, k = torch.zeros(1, Tq, H, 128, device='cuda').bfloat16(), torch.zeros(1, Tk, 1, 128, device='cuda').bfloat16()\n"
            "    lse = A.flash_fwd(q, k, k, 1.0, False)[1].double()\n"
            "    print(float((lse - math.log(Tk)).min()), float((lse - math.log(Tk)).max()))\n")
    env = {k: v for k, v in os.environ.items() if k != "CPB_FWD_POLY"}
    env.update({} if poly is None else {"CPB_FWD_POLY": poly}, PYTHONPATH=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    r = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    values = [float(x) for x in r.stdout.split()]
    assert len(values) == 4
    for v in values:                                        # LSE up to 9.01: fp32 steps of 1e-6, log2 and the sum a few of them
        assert abs(v + share * 7.24e-5) < 4e-6, values


# rows held by one, two, five and eight CTAs, padded columns, an ignored row; the other kernel: a row too wide for a cluster, and
# many rows that L2 holds
@pytest.mark.parametrize("rows,V,Vc", [(5, 17, 64), (3, 26621, 26624), (2, 50257, 50304), (2, 128256, 128256), (2, 212000, 212992), (2, 220000, 220032), (1200, 27001, 27008)])
def test_xent_row_widths(rows, V, Vc):
    from context_parallelism_b200.ops import xent as X
    torch.manual_seed(3)
    lg = torch.randn(rows, Vc, device=dev()) * 4
    tg = torch.randint(0, V, (rows,), device=dev())
    tg[0], tg[1] = V - 1, -100
    loss, row_loss = torch.zeros(1, device=dev()), torch.empty(rows, device=dev())
    d = X.xent_chunk(lg, tg, loss, 0.25, True, row_loss, V)
    check_status()
    x = lg[:, :V].double().requires_grad_()
    want = torch.nn.functional.cross_entropy(x, tg, ignore_index=-100, reduction="none")
    want.sum().backward()
    # fp32 exponentials and sums: 2^-21 relative in the sum, absolute in the loss (values up to 30)
    assert float((row_loss.double() - want).abs().max()) < 2e-5
    assert abs(float(loss) - float(want.sum())) < 2e-5 * rows
    g = torch.zeros(rows, Vc, device=dev(), dtype=torch.float64)
    g[:, :V] = x.grad * 0.25
    assert float((d.double() - g).abs().max()) <= 0.25 * 2.0 ** -8               # one rounding to bf16 of a value below 0.25
    assert float((d.double() - g).norm() / g.norm()) < 2.0 ** -8
    assert bool((d[1] == 0).all()) and bool((d[:, V:] == 0).all())


# widths around the sizes at which a row changes hands (32, 64, 128, 256, 512 threads), rows that leave a turn of four unfinished
@pytest.mark.parametrize("layer", [0, 1])
@pytest.mark.parametrize("rows,d", [(1, 8), (5, 256), (1001, 264), (37, 512), (6, 520), (3, 1024), (2, 1032), (700, 2048), (9, 2056), (4, 4096)])
def test_norm_bwd_widths(layer, rows, d):
    from context_parallelism_b200 import _native as nv
    torch.manual_seed(4)
    x, dy, dr = (torch.randn(rows, d, device=dev()).bfloat16() for _ in range(3))
    w = torch.randn(d, device=dev())
    mean = x.float().mean(1) if layer else torch.zeros(rows, device=dev())
    rstd = torch.rsqrt(((x.float() - mean[:, None]) ** 2).mean(1) + 1e-5)
    stats, dx = torch.stack([mean, rstd], 1).contiguous(), torch.empty_like(x)
    dw, db = torch.ones(d, device=dev()), torch.ones(d, device=dev())
    nv.call("norm_bwd", nv.ptr(x), nv.ptr(dy), nv.ptr(dr), nv.ptr(w), nv.ptr(stats), nv.ptr(dx), nv.ptr(dw), nv.ptr(db if layer else None),
            nv.i(rows), nv.i(d), nv.i(layer), nv.stream_ptr(dev()))
    check_status()
    xh = (x.double() - mean.double()[:, None]) * rstd.double()[:, None]
    g = dy.double() * w.double()
    want = rstd.double()[:, None] * (g - xh * (g * xh).mean(1, keepdim=True) - (g.mean(1, keepdim=True) if layer else 0)) + dr.double()
    assert float((dx.double() - want).norm() / want.norm()) < 2.0 ** -8            # one rounding to bf16
    # fp32 sums over the rows: rows + 4 roundings of 2^-24 of the sum of magnitudes
    for got, term in ((dw, dy.double() * xh), (db, dy.double())) if layer else ((dw, dy.double() * xh),):
        bound = (term.abs().sum(0) + 1) * (rows + 8) * 2.0 ** -24 + 1e-12
        assert bool(((got.double() - 1 - term.sum(0)).abs() <= bound).all())


@pytest.mark.parametrize("layer", [0, 1])
@pytest.mark.parametrize("offset", [0, 1, 4])
def test_norm_bwd_gradient_buffers_at_any_address(layer, offset):
    """Weight gradients of wide rows are added four columns at a time where the buffer is 16-byte aligned, else one at a time."""
    from context_parallelism_b200 import _native as nv
    torch.manual_seed(6)
    rows, d = 70, 1032
    x, dy = (torch.randn(rows, d, device=dev()).bfloat16() for _ in range(2))
    w, stats, dx = torch.randn(d, device=dev()), torch.rand(rows, 2, device=dev()), torch.empty_like(x)
    buf = torch.zeros(2, d + 8, device=dev())
    dw, db = buf[0, offset:], buf[1, offset:]
    nv.call("norm_bwd", nv.ptr(x), nv.ptr(dy), nv.ptr(None), nv.ptr(w), nv.ptr(stats), nv.ptr(dx), nv.ptr(dw), nv.ptr(db if layer else None),
            nv.i(rows), nv.i(d), nv.i(layer), nv.stream_ptr(dev()))
    check_status()
    xh = (x.double() - (stats[:, :1].double() if layer else 0)) * stats[:, 1:].double()
    for got, term in ((dw, dy.double() * xh), (db, dy.double())) if layer else ((dw, dy.double() * xh),):
        # fp32 sums over the rows: rows + 8 roundings of 2^-24 of the sum of magnitudes; nothing beside the d columns is touched
        assert bool(((got[:d].double() - term.sum(0)).abs() <= term.abs().sum(0) * (rows + 8) * 2.0 ** -24 + 1e-12).all())
        assert not bool(got[d:].any())
    assert not bool(buf[:, :offset].any())
