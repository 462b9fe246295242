"""What decides whether a call may be recorded, without a GPU."""
import pytest
import torch

from context_parallelism_b200 import graphs


@pytest.mark.parametrize("where,name", [(torch._C, "_len_torch_dispatch_stack"), (torch._C, "_len_torch_function_stack"),
                                        (torch._C._functorch, "peek_interpreter_stack"), (torch._C._autograd, "_top_saved_tensors_default_hooks"),
                                        (torch.autograd.forward_ad, "_current_level")])
def test_a_torch_without_a_private_name(monkeypatch, where, name):
    """Nothing is recorded then, and nothing raises."""
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    assert graphs._plain_call()
    monkeypatch.delattr(where, name)
    if hasattr(graphs, "_LISTENERS"):                                # resolved at import
        monkeypatch.setattr(graphs, "_LISTENERS", graphs._listeners())
    assert graphs._plain_call() is False


@pytest.mark.parametrize("what", ["head of its own", "one block more", "fewer rows", "transposed", "bias dropped"])
def test_weights_that_changed(what):
    """A record holds for the modules and parameters it was made with: none more, none less, each with its shape and order."""
    from context_parallelism_b200.config import Config
    from context_parallelism_b200.graphs import Weights
    from context_parallelism_b200.models.gpt2 import GPT2
    cfg = Config.from_env("gpt2", 1, env={}).replace(n_embd=64, n_layer=2, n_head=1, n_kv_head=1, head_dim=64, ffn_hidden=256, vocab_size=256, T=32,
                                                      weight_tying=True)
    m = GPT2(cfg)
    w = Weights(m, False)
    assert w.hold()
    if what == "head of its own":
        m.lm_head = torch.nn.Parameter(torch.zeros_like(m.wte))
    elif what == "one block more":
        m.blocks.append(m.blocks[0])
    elif what == "fewer rows":
        m.wte.data = m.wte.data[:128]
    elif what == "transposed":
        m.blocks[1].attn_proj_w.data = m.blocks[1].attn_proj_w.data.t()
    else:
        m.blocks[0].c_fc_b = None
    assert not w.hold()
