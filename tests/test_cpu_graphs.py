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
