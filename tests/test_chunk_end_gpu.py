"""A finished chunk entering the memories of a decode: one kernel per layer against the FP64 definition."""
import pytest
import torch

from warpstate_ai_b200.ops import _ext

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,heads", [(1, 1), (3, 4), (64, 32)])
def test_chunk_end(batch, heads):
    _ext.require()
    torch.manual_seed(batch)
    k, u = (torch.randn(batch, heads, 128, 64, device="cuda").bfloat16() for _ in range(2))
    fast, slow = (torch.randn(batch, heads, 64, 64, device="cuda") for _ in range(2))
    mixed = torch.full((batch, heads, 64, 64), float("nan"), device="cuda", dtype=torch.bfloat16)
    df, ds, mix = (torch.rand(1, heads, 1, 1, device="cuda") for _ in range(3))
    write = torch.tanh(k.double()).transpose(-1, -2) @ torch.tanh(u.double()) / 128
    want_fast, want_slow = df * fast.double() + (1 - df) * write, ds * slow.double() + (1 - ds) * write
    torch.ops.ws_b200.decode_chunk_end(k, u, fast, slow, mixed, df, ds, mix)
    rel = lambda a, b: float((a.double() - b).norm() / b.norm())
    # tanh.approx: 2^-11 per factor, independent over the 128 positions; the memories themselves are FP32
    assert rel(fast, want_fast) < 1e-4 and rel(slow, want_slow) < 1e-4
    assert rel(mixed, mix * want_fast + (1 - mix) * want_slow) < 0.004          # BF16
