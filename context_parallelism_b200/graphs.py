"""CUDA graphs of launch-bound calls: a micro-batch of training, the hidden states or the per-token NLL of a window.

A small model's forward and backward pass is some hundred kernels of 3 to 30 us each, and issuing one costs 13 to 25 us of
Python, autograd and ``ctypes``.  :class:`GraphCache` runs a call eagerly the first times that it sees its shapes, then records it
once and replays the record.  Nothing depends on the caller's buffers: inputs are copied into the record's own, results are
returned as new tensors.  What the record does read by address (weights, gradient buffers) is compared at every call, and a
record whose weights have moved or changed their shape is dropped.  A model's records share one pool of memory; ``CP_GRAPH_POOL_MB`` bounds it, 0 turns records
off.  Measured on one B200, ms without and with records (and without the host's wait for every
micro-batch): next-token logits of 136 tokens, GPT-2 124M 2.69 and 0.71; NLL of 4096 tokens, 48M 1.48 and 0.77; a step of GPT-2 44M, 16
micro-batches of 4 x 1024 tokens 47.7 and 22.6; of GPT-2 124M, two micro-batches 17.6 and 14.9.
"""
from __future__ import annotations

import ctypes
import threading
import weakref
from collections import OrderedDict
from typing import Callable, Optional, Sequence, Tuple

import torch
from torch.autograd import forward_ad

from . import _native as nv

MAX_RECORDS = 32                 # per model; the one used longest ago makes room
# Of the calls with new shapes, the one that is recorded (those before it run as they always did); twice as late each time that the record
# was lost.  A record costs 3 to 30 ms, its launches and 0.3 ms for each block of memory that the driver is asked for: a micro-batch of the 48M
# model 18, 13 of them on top of an eager call, what five replays save.  At the second call a step of two would pay for it in its first pass.
RECORD_AT = 3
MAX_POOL_BYTES = 4 << 30         # buffers of all records of a model, unless its configuration says otherwise (graph_pool_mb)
MIN_FREE_SHARE = 0.25            # share of the GPU's memory that has to be free before a record is made
# A call is recorded while the GPU needs less time for it than the host: a launch costs the host about 25 us (forward and backward;
# 13 us without autograd), the kernels of such models reach about 600 TFLOP/s.
HOST_US_PER_LAUNCH = 25.0
GPU_TFLOPS = 600.0


def model_flops(cfg, batch: int, T: int, train: bool) -> float:
    """Matrix products of one pass over ``batch`` x ``T`` tokens (causal attention; the head at every token)."""
    d, qw = cfg.n_embd, cfg.n_head * cfg.head_dim
    layer = d * (cfg.n_head + 2 * cfg.n_kv_head) * cfg.head_dim + qw * d + (3 if cfg.family == "llama" else 2) * d * cfg.ffn_hidden
    tokens = batch * T
    fwd = 2.0 * tokens * (cfg.n_layer * layer + d * cfg.vocab_size) + 2.0 * batch * T * T * qw * cfg.n_layer
    return (3.3 if train else 1.0) * fwd


class Written:
    """The methods of a model, its blocks and its attention as this package wrote them.  A record runs no Python, so one that holds for
    anything else (a subclass's method, one replaced on a class or an object, another attention) would leave out what that does."""

    def __init__(self, model_cls, block_cls, attn_cls):
        self.model_cls, self.block_cls, self.attn_cls = model_cls, block_cls, attn_cls
        self.methods = {cls: {n: cls.__dict__[n] for n in names} for cls, names in (
            (model_cls, ("hidden", "_hidden", "_block", "head_weight", "loss_with", "loss_sum", "per_token_nll", "recorded_inputs")),
            (block_cls, ("pre_attention", "post_attention")), (attn_cls, ("__call__",)))}

    def _holds(self, cls, obj) -> bool:
        methods = self.methods[cls]
        return isinstance(obj, cls) and _are(type(obj), methods) and methods.keys().isdisjoint(obj.__dict__)

    def model_holds(self, model) -> bool:
        """The model's own methods alone: enough before a replay, in front of which a record looks at the rest (see Weights)."""
        return self._holds(self.model_cls, model)

    def holds(self, model) -> bool:
        attn = model.__dict__.get("attn")
        return (type(attn) is self.attn_cls and attn.ctx.cp_size == 1 and _are(self.attn_cls, self.methods[self.attn_cls])
                and self.model_holds(model) and all(self._holds(self.block_cls, b) for b in model.blocks))

    def of(self, obj):
        """The methods that count for one module of the model."""
        return next((m for cls, m in self.methods.items() if isinstance(obj, cls)), {})


def _are(cls, methods) -> bool:
    for n, f in methods.items():
        if getattr(cls, n, None) is not f:
            return False
    return True


def _read(module) -> tuple:
    """What a record reads of a module beside its parameters: a configuration, which does not change, and an attention's, with its scale."""
    d = module.__dict__
    if "attn" not in d:
        return (d.get("cfg"),)
    attn = d["attn"]
    return d.get("cfg"), getattr(attn, "cfg", attn), type(attn), getattr(attn, "scale", None), getattr(getattr(attn, "ctx", None), "cp_size", 1)


def _listeners():
    """What only private names of torch tell about who is listening; None where one is missing, and nothing is recorded then."""
    try:
        forward_ad._current_level
        return (torch._C._len_torch_dispatch_stack, torch._C._len_torch_function_stack, torch._C._functorch.peek_interpreter_stack,
                torch._C._autograd._top_saved_tensors_default_hooks)
    except AttributeError:
        return None


_LISTENERS = _listeners()


def _plain_call() -> bool:
    """Whether nothing is listening that a replay would pass by: a capture, a mode, a tracer, saved-tensor hooks, a launch timer."""
    if _LISTENERS is None:
        return False
    dispatch_modes, function_modes, transforms, saved_tensor_hooks = _LISTENERS
    return not (torch.cuda.is_current_stream_capturing() or nv._PROFILE is not None or torch.is_anomaly_enabled()
                or dispatch_modes() or function_modes() or transforms() is not None or torch.jit.is_tracing()
                or saved_tensor_hooks(True) is not None or forward_ad._current_level >= 0)


def _main_grad(p) -> int:
    mg = getattr(p, "main_grad", None)
    return 0 if mg is None else mg.data_ptr()


def _quiet(p) -> bool:
    """Whether nobody is to be told about the gradient of ``p``."""
    return getattr(p, "_grad_ready", None) is None and not p._backward_hooks and not p._post_accumulate_grad_hooks


def _unchanged(a: tuple, b: tuple) -> bool:
    return a[0] is b[0] and len(a) == len(b) and (len(a) == 1 or (a[1] is b[1] and a[2:] == b[2:]))


def _NONE():
    """In the place of a weak reference to a module or parameter that is not there."""


class Weights:
    """The modules, their methods and the parameters of a model as a record has them (weak references: a record does not keep its
    model alive)."""

    def __init__(self, model: torch.nn.Module, train: bool, written: Optional[Written] = None):
        self.train = train
        self.mods, self.types = [], {}
        for m in model.modules():
            methods = {} if written is None else written.of(m)
            if methods:
                self.types[type(m)] = methods
            parts = [(n, _NONE if c is None else weakref.ref(c)) for n, c in m._modules.items()]
            params = [(n, weakref.ref(p), p.data_ptr(), p.shape, p.is_contiguous(), _main_grad(p)) if p is not None else (n, _NONE, 0, None, True, 0)
                      for n, p in m._parameters.items()]
            self.mods.append((weakref.ref(m), type(m), methods.keys(), parts, _read(m), params))
        if written is not None:
            self.types[written.attn_cls] = written.methods[written.attn_cls]

    @staticmethod
    def recordable(model: torch.nn.Module) -> bool:
        """A training record needs every gradient in its ``main_grad``."""
        return all(p.requires_grad and _main_grad(p) and _quiet(p) for p in model.parameters())

    def hold(self) -> bool:
        train = self.train
        for cls, methods in self.types.items():
            if not _are(cls, methods):
                return False
        for ref, cls, names, parts, read, params in self.mods:
            m = ref()
            if m is None or type(m) is not cls or not names.isdisjoint(m.__dict__) or not _unchanged(_read(m), read):
                return False
            d = m._modules                                           # one more is a change as well, as is one where there was none
            if len(d) != len(parts):
                return False
            for n, c in parts:
                if n not in d or d[n] is not c() or (d[n] is None and c is not _NONE):
                    return False
            d = m._parameters
            if len(d) != len(params):
                return False
            for n, r, at, shape, dense, grad in params:
                p = d.get(n)
                if p is None:                                        # and was none: a weak reference to what is gone gives None, too
                    if r is not _NONE or n not in d:
                        return False
                    continue
                if p is not r():
                    return False
                if p.data_ptr() != at or p.shape != shape or p.is_contiguous() != dense:
                    return False
                if train and not (p.requires_grad and _main_grad(p) == grad and _quiet(p)):
                    return False
        return True


class _Room:
    """Where the records of a model are made and run: a stream for captures, a pool of memory and the end of the last replay.  Replays
    run one after the other and their results are copied out, so all records of a model work in the same memory."""

    def __init__(self, device: torch.device):
        self.device = device
        self.stream = torch.cuda.Stream(device=device)
        self.pool = torch.cuda.MemPool()
        self.done = torch.cuda.Event()

    def bytes(self) -> int:
        return sum(seg["total_size"] for seg in self.pool.snapshot())

    def short(self) -> bool:
        """Whether less of the GPU's memory is free, or kept by torch for the next allocation, than a record is made with."""
        free, total = torch.cuda.mem_get_info(self.device)
        if free < MIN_FREE_SHARE * total:
            free += torch.cuda.memory_reserved(self.device) - torch.cuda.memory_allocated(self.device) - self.bytes()
        return free < MIN_FREE_SHARE * total


class _Record:
    def __init__(self, fn: Callable, inputs: Sequence[torch.Tensor], weights: Weights, room: _Room):
        """Records ``fn(*inputs)``; nothing is executed.  Raises what ``fn`` or the capture raises."""
        self.weights, self.room = weights, room
        self.exec = ctypes.c_void_p()
        stream = torch.cuda.current_stream(room.device)
        stream.wait_event(room.done)
        with torch.inference_mode(False):
            self.inputs = [torch.zeros(t.shape, dtype=t.dtype, device=room.device) for t in inputs]
        room.done.record(stream)
        lib, launches = nv.lib(), nv.LAUNCHES[0]
        # the backward pass runs in this thread: the pool and the capture are this thread's
        with torch.cuda.stream(room.stream), torch.cuda.use_mem_pool(room.pool), torch.autograd.set_multithreading_enabled(False):
            nv.check(lib.cpb_graph_begin(room.stream.cuda_stream), "graph_begin")
            try:
                outs = fn(*self.inputs)
            except BaseException:
                lib.cpb_graph_end(room.stream.cuda_stream, None)
                raise
            finally:
                self.launches = nv.LAUNCHES[0] - launches
                nv.LAUNCHES[0] = launches
            nv.check(lib.cpb_graph_end(room.stream.cuda_stream, ctypes.byref(self.exec)), "graph_end")
        self.outputs = [o.detach() for o in outs]

    def replay(self, inputs: Sequence[torch.Tensor], stream: torch.cuda.Stream) -> Tuple[torch.Tensor, ...]:
        stream.wait_event(self.room.done)                            # the last replay may have run on another stream
        for s, t in zip(self.inputs, inputs):
            s.copy_(t, non_blocking=True)
        nv.check(nv.lib().cpb_graph_launch(self.exec, stream.cuda_stream, stream.device_index), "graph_launch")
        nv.LAUNCHES[0] += self.launches
        outs = tuple(o.clone() for o in self.outputs)
        self.room.done.record(stream)
        return outs

    def close(self) -> None:
        if self.exec:
            self.room.done.synchronize()                             # the buffers may not be given back under a running replay
            self.outputs = None
            nv.lib().cpb_graph_free(self.exec)
            self.exec = None

    def __del__(self):
        try:
            self.close()
        except Exception:                                            # the end of the process
            pass


class GraphCache:
    """The records of one model, by name, input shapes and modes.  Safe with several threads and streams: a lock covers the copies in,
    the replay and the copies out, and an event orders replays of different streams.  ``limit``: bytes that the records' buffers may
    take together, 0 to record nothing.  ``written``: what the model has to call for a call to be recorded."""

    def __init__(self, limit: int = MAX_POOL_BYTES, written: Optional[Written] = None):
        self.limit, self.written = limit, written
        self._lock = threading.Lock()
        self._room: Optional[_Room] = None                           # there while there are records
        self._records: "OrderedDict[tuple, Optional[_Record]]" = OrderedDict()
        self._seen: "OrderedDict[tuple, tuple]" = OrderedDict()      # eager calls since the record was lost, or at all; launches of one
        self._lost: "OrderedDict[tuple, int]" = OrderedDict()        # how often it was

    def __reduce__(self):                                            # a copied or unpickled model starts without records
        return GraphCache, (self.limit, self.written)

    def __deepcopy__(self, memo):
        return GraphCache(self.limit, self.written)

    def run(self, name: str, model: torch.nn.Module, fn: Callable, inputs: Sequence[torch.Tensor], device: torch.device,
            flops: float, train: bool = False) -> Tuple[torch.Tensor, ...]:
        """``fn(*inputs)`` with the inputs on ``device``: a tuple of tensors."""
        if device.type != "cuda" or self.limit <= 0 or not _plain_call() or any(t.requires_grad for t in inputs):
            return self._eager(fn, inputs, device, train)
        from .ops import attention
        key = (name, device.index, train, torch.is_inference_mode_enabled(), attention.FP32_ACCURATE,
               *((t.dtype, tuple(t.shape)) for t in inputs))
        with self._lock:
            rec = self._records.get(key)
            if rec is not None:
                if rec.weights.hold():
                    self._records.move_to_end(key)
                    return rec.replay(inputs, torch.cuda.current_stream(device))
                self._drop(key)
        if self.written is not None and not self.written.holds(model):
            return self._eager(fn, inputs, device, train)
        with self._lock:
            n, launches = self._seen.get(key, (0, 0))
            if key not in self._records and n + 1 >= RECORD_AT << min(self._lost.get(key, 0), 8):
                self._seen.pop(key, None)
                rec = self._record(key, model, fn, inputs, device, flops < GPU_TFLOPS * 1e6 * HOST_US_PER_LAUNCH * launches, train)
                if rec is not None:
                    return rec.replay(inputs, torch.cuda.current_stream(device))
        before = nv.LAUNCHES[0]
        outs = self._eager(fn, inputs, device, train)
        with self._lock:
            if key not in self._records:
                self._seen[key] = self._seen.pop(key, (0, 0))[0] + 1, nv.LAUNCHES[0] - before
                while len(self._seen) > 64:
                    self._seen.popitem(last=False)
        return outs

    def _eager(self, fn, inputs, device, train: bool):
        """The call without a record.  The records' memory is given back when it runs short: before a backward pass, which cannot be run
        again once it has added to the gradients, and when a forward pass has found no memory."""
        call = lambda: tuple(fn(*(t if t.device == device else t.to(device, non_blocking=True) for t in inputs)))      # noqa: E731
        room = self._room
        if room is None:
            return call()
        if train:
            if room.short():
                with self._lock:
                    self._drop_all()
            return call()
        try:
            return call()
        except torch.OutOfMemoryError:
            pass
        with self._lock:
            self._drop_all()
        return call()

    def _record(self, key, model, fn, inputs, device, launch_bound: bool, train: bool) -> Optional[_Record]:
        free, total = torch.cuda.mem_get_info(device) if launch_bound else (0, 1)
        rec = None
        if free > MIN_FREE_SHARE * total and (not train or Weights.recordable(model)):
            if self._room is None or self._room.device != device:
                self._drop_all()
                self._room = _Room(device)
            try:
                rec = _Record(fn, inputs, Weights(model, train, self.written), self._room)
            except (RuntimeError, nv.NativeError):                   # out of memory, or something in fn that cannot be recorded
                nv.lib().cpb_clear_error()                           # nothing has run; this call and its like are eager
            if rec is not None and self._room.bytes() > self.limit:
                rec.close()
                rec = None
                self._drop_all()
        self._records[key] = rec                                     # None: not to be tried again
        while True:
            held = [k for k, r in self._records.items() if r is not None]
            if len(held) > MAX_RECORDS:
                self._drop(held[0])
            elif len(self._records) > 128:
                self._drop(next(iter(self._records)))
            else:
                break
        if not held:
            self._room = None
        return self._records.get(key)

    def _drop(self, key) -> None:
        rec = self._records.pop(key)
        if rec is not None:
            rec.close()
            self._lost[key] = self._lost.pop(key, 0) + 1
            while len(self._lost) > 64:
                self._lost.popitem(last=False)
            if all(r is None for r in self._records.values()):
                self._room = None

    def _drop_all(self) -> None:
        for key in [k for k, r in self._records.items() if r is not None]:
            self._drop(key)

    def clear(self) -> None:
        """Give back every record and its memory."""
        with self._lock:
            self._drop_all()
            self._records.clear()
            self._seen.clear()
            self._lost.clear()
