"""GEMM tiles of 192 columns and bf16 results split along K: every operand order and epilogue at the edges of the tiles."""
import pytest
import torch

from util import assert_close

pytestmark = pytest.mark.gpu

# Rows and K are chosen so that the plan takes 192 columns: whole tiles, a last tile of 8 and of 184 columns, less than one tile;
# K below one block, with a remainder and over more blocks than the ring of stages holds.
SHAPES = [(256 * 74, 192, 64), (256 * 74, 384, 72), (256 * 37, 376, 520), (4096, 768, 3072), (256 * 74 - 120, 184, 328)]


# 384 columns: two products of 256 and 128 columns per step, one accumulator; M and K with remainders, one and several items per pair
WIDE = [(256 * 74, 384, 2048), (256 * 80 - 120, 384, 2056), (4096, 384, 12008)]


def _operands(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a, b = (torch.randn(r, K, device="cuda", generator=g).bfloat16() for r in (M, N))
    return a, b, torch.randn(N, device="cuda", generator=g), (a.double() @ b.double().t()).float()


@pytest.mark.parametrize("M,N,K", SHAPES + WIDE)
def test_every_epilogue_and_order(M, N, K):
    from context_parallelism_b200 import _native as nv
    from context_parallelism_b200.ops import gemm as G
    a, b, bias, ref = _operands(M, N, K)
    plans = {e: nv.lib().cpb_gemm_plan(M, N, K, e, 0) >> 16 for e in (G.EPI_BF16, G.EPI_F32, G.EPI_F32_ACC, G.EPI_BF16_GELU)}
    assert (384 if (M, N, K) in WIDE else 192) in plans.values(), plans
    at, bt = a.t().contiguous(), b.t().contiguous()
    fp32 = 1e-4 * K ** 0.5                       # two orders of K products of unit normals, see the other GEMM tests
    for x, xm in ((a, False), (at, True)):
        for y, ym in ((b, False), (bt, True)):
            got = G.gemm(x, y, a_mn=xm, b_mn=ym, bias=bias)
            assert_close(got.float(), ref + bias, cos=0.99999, rel=2 ** -8, name=f"bf16 {xm} {ym}")
            assert torch.equal(got, G.gemm(x, y, a_mn=xm, b_mn=ym, bias=bias))
            assert float((G.gemm(x, y, a_mn=xm, b_mn=ym, out_dtype=torch.float32) - ref).abs().max()) < fp32
            acc = torch.ones(M, N, device="cuda")
            G.gemm(x, y, a_mn=xm, b_mn=ym, out=acc, accumulate=True)
            assert float((acc - 1 - ref).abs().max()) < fp32
    pre = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    act = G.gemm(a, b, bias=bias, epi=G.EPI_BF16_GELU, aux=pre)
    assert_close(pre.float(), ref + bias, cos=0.99999, rel=2 ** -8, name="gelu pre")
    assert_close(act.float(), torch.nn.functional.gelu((ref + bias).double(), approximate="tanh").float(), cos=0.99999, rel=2 ** -8, name="gelu")
    nv.status_for(a.device).check("gemm")


# one and two pair-rows, N of one tile and with a remainder, K with a remainder and ranges of unequal length
@pytest.mark.parametrize("M,N,K", [(8, 264, 50304), (136, 768, 3072), (264, 392, 12008), (4096, 384, 50304)])
def test_bf16_split_along_k(M, N, K):
    from context_parallelism_b200 import _native as nv
    from context_parallelism_b200.ops import gemm as G
    assert G.acc_splits(M, N, K, G.EPI_BF16) > 1
    a, b, bias, ref = _operands(M, N, K)
    one = nv.lib().cpb_gemm_plan(M, N, K, G.EPI_F32, 0) & 0xffff
    assert one == 1
    for out in (None, torch.full((M, N + 24), 7.0, device="cuda").bfloat16()):            # dense, and rows of a wider buffer
        dst = None if out is None else out[:, 8:8 + N]
        got = G.gemm(a, b, bias=bias, out=dst)
        whole = G.gemm(a, b, bias=bias, out_dtype=torch.float32)                         # one range of K, not rounded
        assert_close(got.float(), ref + bias, cos=0.99999, rel=2 ** -8, name="split")
        assert float((got.float() - whole.bfloat16().float()).norm() / whole.norm()) < 1e-3      # few values round the other way
        assert torch.equal(got, G.gemm(a, b, bias=bias))
        if out is not None:
            assert bool((out[:, :8] == 7).all() and (out[:, 8 + N:] == 7).all())
    nv.status_for(a.device).check("gemm")


# 384 columns for less than 384: one column of tiles of the next width on, with remainders in M, N and K; two full waves
NARROWER = [(256 * 148 - 120, 384, 4104), (256 * 74 - 8, 264, 2056), (4096, 328, 12008)]


@pytest.mark.parametrize("M,N,K", NARROWER)
def test_one_column_of_384(M, N, K, monkeypatch):
    monkeypatch.setitem(globals(), "WIDE", NARROWER)
    test_every_epilogue_and_order(M, N, K)
