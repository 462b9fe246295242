"""What the language-model head refuses before a launcher gets an address (the launchers see neither types nor widths), without a GPU."""
import pytest
import torch

from context_parallelism_b200 import _native as nv
from context_parallelism_b200.ops import gemm as G
from context_parallelism_b200.ops import xent


class _OnGpu(torch.Tensor):
    """Host memory that takes the GPU's branches."""
    is_cuda = property(lambda self: True)


def _t(*shape, dtype=torch.bfloat16):
    return torch.zeros(shape, dtype=dtype).as_subclass(_OnGpu)


class _Status:
    @staticmethod
    def ptr():
        return 0


@pytest.fixture
def calls(monkeypatch):
    made = []
    monkeypatch.setattr(nv, "call", lambda name, *a: made.append(name))
    monkeypatch.setattr(nv, "status_for", lambda dev: _Status)
    monkeypatch.setattr(nv, "stream_ptr", lambda dev=None: 0)
    return made


@pytest.mark.parametrize("grad", [False, True])
@pytest.mark.parametrize("entry", [xent.per_token_nll, xent.linear_cross_entropy])
@pytest.mark.parametrize("x,w,rows", [
    ((6, 64, torch.float32), (16, 64, torch.bfloat16), 6), ((6, 64, torch.bfloat16), (16, 64, torch.float32), 6),
    ((6, 64, torch.float16), (16, 64, torch.float16), 6), ((6, 64, torch.bfloat16), (16, 56, torch.bfloat16), 6),
    ((6, 64, torch.bfloat16), (16, 72, torch.bfloat16), 6), ((6, 64, torch.bfloat16), (16, 64, torch.bfloat16), 5)])
def test_refused_before_a_launch(calls, entry, x, w, rows, grad):
    a, b = _t(*x[:2], dtype=x[2]), _t(*w[:2], dtype=w[2])
    if grad:
        a.requires_grad_()
    with pytest.raises(AssertionError):
        entry(a, b, torch.zeros(rows, dtype=torch.int64))
    assert not calls


def test_refused_on_another_device(calls):
    with pytest.raises(AssertionError):
        xent.per_token_nll(_t(6, 64), torch.zeros(16, 64, dtype=torch.bfloat16, device="meta"), torch.zeros(6, dtype=torch.int64))
    assert not calls


@pytest.mark.parametrize("tdtype", [torch.int32, torch.int64])
def test_accepted(calls, tdtype):
    assert xent.per_token_nll(_t(2, 3, 64), _t(16, 64), torch.zeros(2, 3, dtype=tdtype)).shape == (6,)
    assert calls == ["gemm_head", "xent_rows"]


def test_rows_at_one_address():
    """Rows that are one row expanded are copied out: a tensor map takes no stride of zero."""
    assert G._rowmajor2d(torch.zeros(1, 64).expand(4, 64)).stride() == (64, 1)
    for keep in (torch.zeros(4, 64), torch.zeros(4, 72)[:, :64], torch.zeros(1, 64)):
        assert G._rowmajor2d(keep).data_ptr() == keep.data_ptr()
