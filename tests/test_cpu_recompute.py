"""Recomputation in the backward pass of a model with a part of the caller's own, without a GPU."""
import pytest
import torch

from context_parallelism_b200.config import Config


@pytest.mark.parametrize("recompute", ["selective", "full"])
@pytest.mark.parametrize("family", ["llama", "gpt2"])
def test_a_block_that_draws_random_numbers(family, recompute):
    """Dropout in a block's method draws the same mask when the part is computed again."""
    from context_parallelism_b200.models.gpt2 import GPT2
    from context_parallelism_b200.models.llama import Llama
    grads = []
    for mode in ("none", recompute):
        cfg = Config.from_env(family, 1, env={}).replace(
            n_embd=64, n_layer=2, n_head=2, n_kv_head=2, head_dim=32, ffn_hidden=128, vocab_size=100, T=16, B=2, dtype="fp32", recompute=mode)
        model = (Llama if family == "llama" else GPT2)(cfg)
        for blk in model.blocks:
            def post(x, o, f=blk.post_attention):
                x, pending = f(x, o)
                return x, torch.nn.functional.dropout(pending, 0.5)
            blk.post_attention = post
        idx = torch.randint(0, 100, (2, 16), generator=torch.Generator().manual_seed(1))
        torch.manual_seed(7)
        model.loss_sum(idx, idx, torch.arange(16)).backward()
        grads.append(torch.cat([p.grad.flatten() for p in model.parameters()]))
    assert torch.allclose(*grads, rtol=1e-4, atol=1e-6)
