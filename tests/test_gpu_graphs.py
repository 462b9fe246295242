"""Recorded calls (``graphs.py``) against the same calls run eagerly: every replay reads the inputs and weights of its own call."""
import copy
import gc
import threading
import weakref

import pytest
import torch

from util import assert_close

pytestmark = pytest.mark.gpu


def _engine(family="llama", recompute="none", **kw):
    from context_parallelism_b200.config import Config
    from context_parallelism_b200.engine import TrainEngine
    cfg = Config.from_env(family, 1, env={}).replace(**{**dict(
        n_embd=256, n_layer=2, n_head=4, n_kv_head=2 if family == "llama" else 4, head_dim=64, ffn_hidden=512 if family == "llama" else 1024,
        vocab_size=1000, T=200, B=2, max_steps=20, warmup_steps=1, checkpointing=False, recompute=recompute, dtype="bf16",
        weight_tying=family == "gpt2"), **kw})
    return TrainEngine(cfg, torch.device("cuda", 0))


def _batch(eng, seed, T=0):
    t = torch.randint(0, eng.cfg.vocab_size, (eng.cfg.B, (T or eng.cfg.T) + 1), generator=torch.Generator().manual_seed(seed))
    return t[:, :-1].contiguous().pin_memory(), t[:, 1:].contiguous().pin_memory()


def _records(eng):
    return [r for r in eng.model.graphs._records.values() if r is not None]


@pytest.mark.parametrize("family,recompute", [("llama", "none"), ("llama", "selective"), ("llama", "full"), ("gpt2", "none"), ("gpt2", "selective")])
def test_micro_batches_and_steps(family, recompute):
    a, b = _engine(family, recompute), _engine(family, recompute)
    b._recordable = lambda *args: False
    for step in range(3):
        for i in range(3):
            la, lb = (e.forward_backward(*_batch(e, 10 * step + i), accum=3, last=i == 2) for e in (a, b))
            assert abs(float(la) - float(lb)) <= 1e-4 * abs(float(lb))
        # dQ, norm, bias and embedding gradients are fp32 sums in arrival order; two eager passes differ as much
        assert_close(a.flat.grad, b.flat.grad, cos=0.99999, rel=1e-2, name="grad")
        a.optimizer_step(), b.optimizer_step()
        b.flat.master.copy_(a.flat.master), b.flat.sync_compute_copy(), b.flat.m.copy_(a.flat.m), b.flat.v.copy_(a.flat.v)
    assert len(_records(a)) == 1 and not _records(b)
    a.check_kernels()


@pytest.mark.parametrize("family", ["llama", "gpt2"])
@torch.no_grad()
def test_forward_calls_are_bit_equal(family):
    from context_parallelism_b200.ops import rope, xent
    eng = _engine(family)
    for i in range(6):
        x, y, pos = eng.shard_batch(*_batch(eng, i, T=136 + 8 * (i % 2)))
        kept = None
        if family == "llama" and i >= 4:                             # another position scaling: a table at another address
            eng.model.set_rope_cache(rope.build_rope_cache(eng.cfg.T, 64, 500.0 + i, eng.device, None))
        if i == 5:
            eng.model.head_weight().data.mul_(1.5)
        for _ in range(2):
            got = eng.model.per_token_nll(x, y, pos), eng.model.hidden(x, pos)
            want_h = eng.model._hidden(x, pos, *eng.model.recorded_inputs())
            want = xent.per_token_nll(want_h, eng.model.head_weight(), y, eng.cfg.vocab_size).view(x.shape), want_h
            assert all(torch.equal(g, w) for g, w in zip(got, want))
            kept = kept or got
        assert all(torch.equal(g, w) for g, w in zip(kept, want))    # a later call does not write into earlier results
    assert len(_records(eng)) == 4


@torch.no_grad()
def test_moved_weights_and_copies():
    eng = _engine()
    x, y, pos = eng.shard_batch(*_batch(eng, 1))
    first = [eng.model.per_token_nll(x, y, pos) for _ in range(3)][-1]
    assert len(_records(eng)) == 1
    old = eng.model.blocks[0].wo
    eng.model.blocks[0].wo = torch.nn.Parameter(old.detach() * 2)
    assert not torch.equal(eng.model.per_token_nll(x, y, pos), first) and not _records(eng)
    eng.model.blocks[0].wo = old
    other = copy.deepcopy(eng.model)
    assert torch.equal(other.per_token_nll(x, y, pos), first) and not other.graphs._records
    eng.close()
    assert not eng.model.graphs._records


def test_what_is_not_recorded():
    """Hooks see every call; an engine is freed without the garbage collector."""
    eng = _engine()
    seen = []
    h = eng.model.norm_f.register_hook(lambda g: seen.append(g))
    for i in range(4):
        eng.forward_backward(*_batch(eng, i))
    assert not _records(eng)
    h.remove()
    eng.model.graphs.clear()
    for i in range(3):
        with torch.autograd.graph.saved_tensors_hooks(lambda t: seen.append(1) or t, lambda t: t):
            eng.forward_backward(*_batch(eng, i))
    assert not _records(eng) and seen
    for i in range(3):
        eng.forward_backward(*_batch(eng, i))
    assert len(_records(eng)) == 1
    eng.check_kernels()
    gc.collect()
    gc.disable()
    try:
        ref = weakref.ref(eng.model)
        del eng, h
        assert ref() is None
    finally:
        gc.enable()


def _replace(eng, what, seen, monkeypatch):
    """Put something that counts its calls in the place of a part of the model; returns how often one forward pass calls it."""
    m = eng.model
    count = lambda f: lambda *a, **k: (seen.append(1), f(*a, **k))[1]          # noqa: E731
    if what == "attention":
        m.attn = count(m.attn)
        return len(m.blocks)
    if what == "subclass":
        m.__class__ = type("Own", (type(m),), {"_hidden": count(type(m)._hidden)})
        return 1
    if what == "block":
        m.blocks[1].pre_attention = count(m.blocks[1].pre_attention)
        return 1
    monkeypatch.setattr(type(m.blocks[0]), "post_attention", count(type(m.blocks[0]).post_attention))
    return len(m.blocks)


@pytest.mark.parametrize("what", ["attention", "subclass", "block", "block class"])
@pytest.mark.parametrize("family", ["llama", "gpt2"])
def test_what_the_caller_put_into_the_model_runs_every_time(family, what, monkeypatch):
    eng, seen = _engine(family), []
    x, y, pos = eng.shard_batch(*_batch(eng, 1))
    per_pass = _replace(eng, what, seen, monkeypatch)
    for grad, call in ((False, lambda: eng.model.hidden(x, pos)), (False, lambda: eng.model.per_token_nll(x, y, pos)),
                       (True, lambda: eng.forward_backward(x, y))):
        del seen[:]
        for _ in range(6):
            with torch.set_grad_enabled(grad):
                call()
        assert len(seen) == 6 * per_pass
    assert not _records(eng)


@torch.no_grad()
def test_another_attention_scale():
    eng = _engine()
    x, _, pos = eng.shard_batch(*_batch(eng, 1))
    first = [eng.model.hidden(x, pos) for _ in range(4)][-1]
    eng.model.attn.scale *= 2
    assert torch.equal(eng.model.hidden(x, pos), eng.model._hidden(x, pos, eng.model.rope_cache))
    eng.model.attn.scale /= 2
    eng.model.attn = type(eng.model.attn)(eng.cfg, eng.cp)           # another object, the same attention
    assert torch.equal(eng.model.hidden(x, pos), first)


@torch.no_grad()
def test_more_shapes_than_records(monkeypatch):
    """Shapes met in turn, one more than there is room for: results stay right, and the records lost are made ever less often."""
    from context_parallelism_b200 import graphs
    monkeypatch.setattr(graphs, "MAX_RECORDS", 2)
    eng, made = _engine(), []
    init = graphs._Record.__init__
    monkeypatch.setattr(graphs._Record, "__init__", lambda self, *a: (made.append(1), init(self, *a))[1])
    batches = [eng.shard_batch(*_batch(eng, i, T=104 + 8 * i)) for i in range(3)]
    want = [eng.model._hidden(x, p, *eng.model.recorded_inputs()) for x, _, p in batches]
    for _ in range(16):
        for (x, _, p), w in zip(batches, want):
            assert torch.equal(eng.model.hidden(x, p), w)
    assert len(_records(eng)) <= 2 and len(made) <= 9


@torch.no_grad()
def test_threads_and_streams():
    from context_parallelism_b200.ops import xent
    eng = _engine()
    batches = [eng.shard_batch(*_batch(eng, i)) for i in range(4)]
    want = [xent.per_token_nll(eng.model._hidden(x, p, *eng.model.recorded_inputs()), eng.model.head_weight(), y, 1000).view(x.shape)
            for x, y, p in batches]
    torch.cuda.synchronize()
    bad = []

    def work(k):
        with torch.no_grad(), torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(12):
                got = eng.model.per_token_nll(*batches[k])
                torch.cuda.current_stream().synchronize()
                if not torch.equal(got, want[k]):
                    bad.append(k)
    ts = [threading.Thread(target=work, args=(k,), daemon=True) for k in range(4)]
    [t.start() for t in ts]
    [t.join(60) for t in ts]
    assert not any(t.is_alive() for t in ts) and not bad and len(_records(eng)) == 1
    eng.check_kernels()


@torch.no_grad()
def test_another_thread_draws_random_numbers_while_one_records():
    eng, stop, raised = _engine(), threading.Event(), []

    def draw():
        with torch.cuda.stream(torch.cuda.Stream()):
            while not stop.is_set():
                try:
                    torch.randn(100, device="cuda")
                except RuntimeError as e:
                    raised.append(str(e))
    t = threading.Thread(target=draw, daemon=True)
    t.start()
    for T in range(64, 128, 8):
        x, _, pos = eng.shard_batch(*_batch(eng, T, T=T))
        want = eng.model._hidden(x, pos, *eng.model.recorded_inputs())
        assert all(torch.equal(eng.model.hidden(x, pos), want) for _ in range(5))
    stop.set()
    t.join(60)
    assert len(_records(eng)) == 8 and not raised and not t.is_alive()


@torch.no_grad()
def test_a_call_that_cannot_be_recorded():
    """A capture that fails leaves the call as it was: eager from then on, its like and everything else usable."""
    from context_parallelism_b200.graphs import GraphCache
    eng, cache = _engine(), GraphCache()
    x, _, pos = eng.shard_batch(*_batch(eng, 1))

    def waits(idx):
        torch.cuda.current_stream().synchronize()                    # not allowed while a stream records
        return (eng.model._hidden(idx, pos, eng.model.rope_cache),)
    want = waits(x)[0]
    for _ in range(5):
        assert torch.equal(cache.run("waits", eng.model, waits, (x,), eng.device, 0.0)[0], want)
        assert torch.equal(eng.model.hidden(x, pos), want)
    assert list(cache._records.values()) == [None] and len(_records(eng)) == 1
    eng.check_kernels()


@torch.no_grad()
def test_records_share_memory_and_give_it_back():
    """Records of different calls in one pool, replayed in turn and on two streams, keep their results apart."""
    eng = _engine(vocab_size=8000)
    cases = [eng.shard_batch(*_batch(eng, i, T=T)) for i, T in enumerate((200, 192, 128))]
    want = [(eng.model._hidden(x, p, *eng.model.recorded_inputs()), eng.model.per_token_nll(x, y, p)) for x, y, p in cases]
    before, other, sizes = torch.cuda.memory_reserved(), torch.cuda.Stream(), []
    torch.cuda.synchronize()
    for i in range(12):
        with torch.cuda.stream(other if i % 2 else torch.cuda.current_stream()):
            got = [(eng.model.hidden(x, p), eng.model.per_token_nll(x, y, p)) for x, y, p in cases]
        torch.cuda.synchronize()
        assert all(torch.equal(g, w) for pair, ref in zip(got, want) for g, w in zip(pair, ref))
        sizes += [eng.model.graphs._room.bytes()] if eng.model.graphs._room else []
    assert len(_records(eng)) == 6 and len({id(r.room) for r in _records(eng)}) == 1
    assert sizes[-1] <= 64 << 20                                     # in pools of their own each would have segments of 2 and 20 MB
    eng.close()
    assert eng.model.graphs._room is None and torch.cuda.memory_reserved() <= before + (40 << 20)


@torch.no_grad()
def test_limit_of_the_records_memory():
    for mb, made in ((0, False), (1, False), (4096, True)):
        eng = _engine(graph_pool_mb=mb)
        x, y, pos = eng.shard_batch(*_batch(eng, 1))
        want = eng.model._hidden(x, pos, *eng.model.recorded_inputs())
        assert all(torch.equal(eng.model.hidden(x, pos), want) for _ in range(5))
        assert bool(_records(eng)) == made == (eng.model.graphs._room is not None)


def test_memory_is_given_back_when_it_runs_short(monkeypatch):
    from context_parallelism_b200 import graphs
    eng, left = _engine(), [1]
    x, y, pos = eng.shard_batch(*_batch(eng, 1))
    with torch.no_grad():
        for _ in range(3):
            eng.model.hidden(x, pos)
        assert len(_records(eng)) == 1

        def full(idx):
            if left:
                left.pop()
                raise torch.OutOfMemoryError("full")
            return (idx + len(_records(eng)),)
        assert torch.equal(eng.model.graphs.run("full", eng.model, full, (x,), eng.device, 0.0)[0], x)          # run again without records
        for _ in range(12):
            eng.model.hidden(x, pos)
        assert len(_records(eng)) == 1
    eng.forward_backward(*_batch(eng, 2))
    assert len(_records(eng)) == 1                                   # memory is plenty
    monkeypatch.setattr(graphs, "MIN_FREE_SHARE", 2.0)
    eng.forward_backward(*_batch(eng, 3))
    assert not _records(eng) and eng.model.graphs._room is None
    eng.check_kernels()


def test_generation_keeps_its_records(monkeypatch):
    """The trainers' generation loop meets each padded length eight times and puts an attention of its own into the model for every call."""
    from context_parallelism_b200 import graphs
    from context_parallelism_b200.trainers.gpt2_cp import generate
    eng, made = _engine("gpt2"), []
    init = graphs._Record.__init__
    monkeypatch.setattr(graphs._Record, "__init__", lambda self, *a: (made.append(1), init(self, *a))[1])
    prompt = torch.randint(0, 1000, (1, 20), generator=torch.Generator().manual_seed(1))
    first, after = generate(eng, prompt, 96), len(made)
    assert after >= 11                                               # lengths of 24 to 120; the record of one that was met twice is not made
    for _ in range(2):
        assert torch.equal(generate(eng, prompt, 96), first)
    assert len(made) <= after + 1
    eng.check_kernels()


@pytest.mark.parametrize("train", [False, True])
def test_the_call_that_is_recorded_is_not_run_eagerly_too(train):
    """Of six calls two run eagerly and the third records and replays: recording on top of an eager call made first passes slower."""
    eng, ran, got = _engine(), [], []
    x, y, pos = eng.shard_batch(*_batch(eng, 1))
    run = eng.model.graphs.run
    eng.model.graphs.run = lambda n, m, fn, *a, **k: run(n, m, lambda *t: (ran.append(1), fn(*t))[1], *a, **k)
    for _ in range(6):
        with torch.set_grad_enabled(train):
            got.append(float(eng.forward_backward(x, y)) if train else eng.model.hidden(x, pos))
    assert len(ran) == 3 and len(_records(eng)) == 1
    assert all(abs(g - got[0]) <= 1e-4 * abs(got[0]) if train else torch.equal(g, got[0]) for g in got)
    eng.check_kernels()
