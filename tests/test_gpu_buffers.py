"""Token buffers that the caller writes to again as soon as a micro-batch has been issued, while the GPU is still busy with earlier work."""
import pytest
import torch

from util import assert_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("recorded", [True, False])
@pytest.mark.parametrize("view", [False, True])
def test_buffers_are_written_again_at_once(recorded, view):
    from context_parallelism_b200.config import Config
    from context_parallelism_b200.engine import TrainEngine
    cfg = Config.from_env("llama", 1, env={}).replace(
        n_embd=256, n_layer=2, n_head=4, n_kv_head=2, head_dim=64, ffn_hidden=512, vocab_size=1000, T=200, B=2, checkpointing=False, dtype="bf16")
    a, b = (TrainEngine(cfg, torch.device("cuda", 0)) for _ in range(2))
    if not recorded:
        a._recordable = lambda *args: False
    b._recordable = lambda *args: False
    batches = [torch.randint(0, 1000, (2, 201), generator=torch.Generator().manual_seed(i)) for i in range(8)]
    # as the loaders have them: two pairs in turn, or two buffers of which tokens and targets are views
    buf = [torch.empty(2, 201, dtype=torch.int64).pin_memory() for _ in range(2)]
    pairs = [(t[:, :-1], t[:, 1:]) if view else (t[:, :-1].contiguous().pin_memory(), t[:, 1:].contiguous().pin_memory()) for t in buf]
    losses = []
    for i, t in enumerate(batches):
        x, y = pairs[i % 2]
        x.copy_(t[:, :-1]), y.copy_(t[:, 1:])
        torch.cuda._sleep(20_000_000)                                # 10 ms: the copies wait behind it
        losses.append(a.forward_backward(x, y, accum=8, last=i == 7))
    want = [b.forward_backward(t[:, :-1].contiguous().cuda(), t[:, 1:].contiguous().cuda(), accum=8, last=i == 7) for i, t in enumerate(batches)]
    for la, lb in zip(losses, want):
        assert abs(float(la) - float(lb)) <= 1e-4 * abs(float(lb))
    assert_close(a.flat.grad, b.flat.grad, cos=0.99999, rel=1e-2, name="grad")
    a.check_kernels()


def test_a_graph_of_the_callers_reads_the_callers_buffers():
    """A capture of a whole micro-batch keeps the caller's page-locked buffers as its inputs."""
    from context_parallelism_b200.config import Config
    from context_parallelism_b200.engine import TrainEngine
    cfg = Config.from_env("llama", 1, env={}).replace(
        n_embd=256, n_layer=2, n_head=4, n_kv_head=2, head_dim=64, ffn_hidden=512, vocab_size=1000, T=200, B=2, checkpointing=False, dtype="bf16")
    eng = TrainEngine(cfg, torch.device("cuda", 0))
    batches = [torch.randint(0, 1000, (2, 201), generator=torch.Generator().manual_seed(i)) for i in range(3)]
    x, y = (torch.zeros(2, 200, dtype=torch.int64).pin_memory() for _ in range(2))
    want = [float(eng.forward_backward(t[:, :-1].contiguous().cuda(), t[:, 1:].contiguous().cuda())) for t in batches]
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        loss = eng.forward_backward(x, y)
    for t, w in zip(batches, want):
        x.copy_(t[:, :-1]), y.copy_(t[:, 1:])
        graph.replay()
        torch.cuda.synchronize()
        assert abs(float(loss) - w) <= 1e-4 * abs(w)
    eng.check_kernels()
