"""What a prefill is made of runs without autograd, whatever the caller's mode: its operators have no backward formula."""
from types import SimpleNamespace

import pytest
import torch

from warpstate_ai_b200 import WarpStateConfig
from warpstate_ai_b200.models.warpstate import WarpStateCore
from warpstate_ai_b200.ops import attention, fused


@pytest.mark.parametrize("last", [False, True])
def test_a_block_with_gradients_enabled(monkeypatch, last):
    core = WarpStateCore(WarpStateConfig(vocab_size=64, d_model=128, n_heads=2, n_cores=1, logical_depth=1, ffn_hidden=64, chunk_size=128,
                                         gradient_checkpointing=False, parallel_memory=True))
    modes = []

    def rows(t, *rest):
        modes.append(torch.is_grad_enabled())
        return t * core.norm1.weight

    monkeypatch.setattr(fused, "_prefill_norm", lambda core, x, scale, bias: (rows(x), rows(x)))
    monkeypatch.setattr(fused, "bf16_weight", lambda p: p)
    monkeypatch.setattr(fused.G, "linear", lambda x, w: rows(x))
    monkeypatch.setattr(attention, "prefill", lambda qkvgu, *rest: rows(qkvgu))
    monkeypatch.setattr(fused, "_prefill_finish", lambda core, y, xmod: rows(y) + xmod)
    with torch.enable_grad():
        out = fused.core_prefill_state(core, torch.randn(6, 128), torch.ones(128), torch.ones(128), 2, 3, SimpleNamespace(), last)
    assert modes and not any(modes)
    assert not any(t.requires_grad for t in (out if last else (out,)))
