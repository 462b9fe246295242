"""Cross entropy in the epilogue of the head's GEMM (``cpb_gemm_head``, ``cpb_xent_rows``) against 64-bit results of the same bf16 operands."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(rows, d, V, n_valid, spread=1.0):
    g = torch.Generator(device="cuda").manual_seed(rows + d + V)
    x = (torch.randn(rows, d, device="cuda", generator=g) * spread).bfloat16()
    w = torch.zeros(V, d, device="cuda")
    w[:n_valid] = torch.randn(n_valid, d, device="cuda", generator=g) / d ** 0.5
    w = w.bfloat16()
    tg = torch.randint(0, n_valid, (rows,), device="cuda", generator=g)
    tg[0], tg[rows // 2] = n_valid - 1, -100
    return x, w, tg


# edges: one row, less and more than a warp's, a CTA's and a pair's rows; columns in one tile, one more than a tile's, a last tile of padding only
@pytest.mark.parametrize("rows,d,V,n_valid,spread", [
    (1, 64, 8, 8, 1), (31, 64, 64, 57, 1), (33, 72, 264, 257, 1), (129, 128, 512, 250, 1), (257, 384, 1024, 1000, 30), (300, 1024, 8192, 8192, 1),
    (4096 + 5, 384, 50304, 50257, 1), (64, 768, 128256, 128256, 8)])
def test_loss_and_dlogits(rows, d, V, n_valid, spread):
    from context_parallelism_b200.ops import xent
    x, w, tg = _case(rows, d, V, n_valid, spread)
    scale = 0.7 / rows
    total, row = torch.zeros(1, device="cuda"), torch.empty(rows, device="cuda")
    coef = xent._head_rows(x, w, tg, n_valid, scale, total, row, True)
    dlog = xent._head_dlogits(x, w, tg, coef, n_valid, scale)
    logits = (x.double() @ w.double().T)[:, :n_valid]
    seen = tg >= 0
    want = torch.where(seen, torch.logsumexp(logits, 1) - logits.gather(1, tg.clamp(min=0)[:, None])[:, 0], 0.0)
    # fp32 sums of d products, then of n_valid exponentials: far below 1e-5 of the largest term
    tol = 1e-5 * (1 + float(logits.abs().max()))
    assert float((row - want).abs().max()) <= tol
    assert abs(float(total) - float(want.sum())) <= tol * rows
    p = torch.softmax(logits, 1)
    p[seen, tg[seen]] -= 1
    p = p * seen[:, None] * scale
    err = (dlog[:, :n_valid].double() - p).abs()
    assert bool((err <= 2 ** -8 * p.abs() + tol * scale).all())            # one rounding to bf16 (2^-9) beside the fp32 error
    assert not bool(dlog[:, n_valid:].any())
    logits32 = torch.full((rows, V + 8), 3.0, device="cuda")[:, :V]
    stored = xent._head_rows(x, w, tg, n_valid, scale, None, row2 := torch.empty_like(row), True, logits32)
    assert torch.equal(row, row2) and torch.equal(coef, stored)
    assert float((logits32[:, :n_valid].double() - logits).abs().max()) <= tol
    other = xent._head_dlogits(x, w, tg, stored, n_valid, scale, logits32)
    assert bool(((other[:, :n_valid].double() - p).abs() <= 2 ** -8 * p.abs() + tol * scale).all()) and not bool(other[:, n_valid:].any())
    again = xent._head_rows(x, w, tg, n_valid, scale, None, row2 := torch.empty_like(row), True)
    assert torch.equal(row, row2) and torch.equal(coef, again)


def test_values_that_are_no_numbers():
    """A NaN or an infinity in a row makes that row's loss NaN and leaves the others alone, as the kernel on stored logits does."""
    from context_parallelism_b200.ops import xent
    x, w, tg = _case(40, 64, 512, 500)
    x[3, 5], x[7, 0] = float("nan"), float("inf")
    row, old = torch.empty(40, device="cuda"), torch.empty(40, device="cuda")
    xent._head_rows(x, w, tg, 500, 1.0, None, row, False)
    logits = xent.gemm(x, w, out_dtype=torch.float32)
    xent.xent_chunk(logits, tg, None, 1.0, False, old, 500)
    assert torch.equal(row.isnan(), old.isnan()) and bool(row[[3, 7]].isnan().all())
    ok = ~row.isnan()
    assert float((row - old)[ok].abs().max()) < 1e-5


@pytest.mark.parametrize("d", [1024, 1032])                                  # both sides of the rule
@pytest.mark.parametrize("rows", [70, 4099])
def test_gradients_on_both_sides_of_the_rule(d, rows):
    from context_parallelism_b200.ops import xent
    assert xent.RECOMPUTE_WIDTH == 1024
    x, w, tg = _case(rows, d, 1024, 1000)
    x.requires_grad_(), w.requires_grad_()
    loss = xent.linear_cross_entropy(x, w, tg, 1.0 / rows, 1000)
    loss.backward(torch.full_like(loss, 1.0 / rows))
    X, W = x.detach().double().requires_grad_(), w.detach().double().requires_grad_()
    want = torch.nn.functional.cross_entropy((X @ W.T)[:, :1000], tg, ignore_index=-100, reduction="sum")
    (want / rows).backward()
    assert abs(float(loss) - float(want)) < 1e-5 * float(want)
    for got, ref in ((x.grad, X.grad), (w.grad, W.grad)):
        # dlogits and the result are each rounded to bf16: 2^-9 relative in norm, both together below 4e-3
        assert float((got.double() - ref).norm() / ref.norm()) < 4e-3
    with torch.no_grad():
        assert abs(float(xent.linear_cross_entropy(x, w, tg, 0.0, 1000)) - float(want)) < 1e-5 * float(want)
