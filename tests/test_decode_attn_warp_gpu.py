"""The decode attention with a warp per (sequence, head), which many of them take, against the kernel with a CTA for each, which few take."""
import pytest
import torch

from warpstate_ai_b200 import WarpStateConfig, WarpStateLM
from warpstate_ai_b200.ops import _ext, attention, gemm
from warpstate_ai_b200.serve.engine import DecodeEngine


# the first row, the edges of the 32 rows that come at a time, the last row; a count that leaves warps of the last CTA idle
@pytest.mark.gpu
@pytest.mark.parametrize("pos", [0, 1, 31, 32, 33, 64, 95, 127])
@pytest.mark.parametrize("batch,heads", [(40, 32), (64, 19), (61, 21)])
def test_a_warp_per_head_gives_what_a_cta_per_head_gives(batch, heads, pos):
    """FP32 sums in another order, then one rounding to BF16: half an ulp of the larger neighbour at most, 2 ** -8 of the value."""
    _ext.require()
    torch.manual_seed(pos + heads)
    ops, d = torch.ops.ws_b200, 64 * heads
    rope, at = attention.rope_table(torch.device("cuda", 0)), torch.tensor(pos, device="cuda")
    qkvgu = (torch.randn(batch, 5 * d, device="cuda") * 1.5).bfloat16()
    state = [torch.randn(batch, heads, 128, 64, device="cuda").bfloat16() for _ in range(3)]
    mixed = torch.randn(batch, heads, 64, 64, device="cuda").bfloat16()
    for cache in state:
        cache[:, :, pos + 1:] = float("nan")               # nothing behind the position may be looked at
    assert batch * heads > 1184

    def step(part, caches):
        y = torch.full((qkvgu[part].shape[0], d), float("nan"), device="cuda", dtype=torch.bfloat16)
        ops.decode_attn(qkvgu[part].contiguous(), *caches, mixed[part].contiguous(), rope, at, heads, y, False)
        return y

    many = [t.clone() for t in state]
    y = step(slice(None), many)
    for first in range(0, batch, 20):                      # at most 640 heads: a CTA for each
        part = slice(first, first + 20)
        few = [t[part].clone() for t in state]
        want = step(part, few)
        assert torch.allclose(y[part].float(), want.float(), rtol=2 ** -7, atol=1e-4)
        assert float((y[part].float() - want.float()).norm() / want.float().norm()) < 1e-3
        for mine, theirs in zip(many, few):
            assert torch.equal(mine[part].view(torch.int16), theirs.view(torch.int16))


@pytest.mark.gpu
def test_outputs_at_any_element():
    """The kernel with a warp per head stores 16 bytes at a time; outputs that begin elsewhere are written by the other one."""
    _ext.require()
    torch.manual_seed(3)
    batch, heads = 40, 32
    ops, d = torch.ops.ws_b200, 64 * heads
    rope, at = attention.rope_table(torch.device("cuda", 0)), torch.tensor(50, device="cuda")
    qkvgu = torch.randn(batch, 5 * d, device="cuda").bfloat16()
    caches = [torch.randn(batch, heads, 128, 64, device="cuda").bfloat16() for _ in range(3)]
    mixed = torch.randn(batch, heads, 64, 64, device="cuda").bfloat16()
    room = torch.zeros(2, batch * d + 8, device="cuda", dtype=torch.bfloat16)
    results = []
    for part, offset in zip(room, (0, 3)):
        y = part[offset:offset + batch * d].view(batch, d)
        ops.decode_attn(qkvgu, *[t.clone() for t in caches], mixed, rope, at, heads, y, False)
        results.append(y.float())
    assert float((results[0] - results[1]).norm() / results[1].norm()) < 1e-3
    assert not room[1, :3].any() and not room[1, 3 + batch * d:].any()


# captured, the step requests the position, the caches and half of the memories ahead of its turn; a count that leaves warps of the last CTA
# idle, over the edges of the 32 rows that come at a time, the end of a chunk and the first rows of the next
@pytest.mark.gpu
@pytest.mark.parametrize("batch,heads", [(40, 32), (41, 29)])
def test_captured_steps_give_what_steps_one_by_one_give(batch, heads):
    torch.manual_seed(heads)
    cfg = WarpStateConfig(vocab_size=512, d_model=64 * heads, n_heads=heads, n_cores=2, logical_depth=2, ffn_hidden=128, chunk_size=128,
                          gradient_checkpointing=False, parallel_memory=True)
    with torch.device("cuda"):
        model = WarpStateLM(cfg).eval().requires_grad_(False)
    assert batch * heads > 1184
    ids = torch.randint(0, 512, (batch, 170), device="cuda")
    captured, single = DecodeEngine(model), DecodeEngine(model, use_cuda_graph=False)
    for position in range(ids.shape[1]):
        got, want = captured.step(ids[:, position]), single.step(ids[:, position])
        assert torch.equal(got, want), position
    gemm.check_device_errors()
    assert captured.graph_counters.replay_calls == ids.shape[1] and single.graph_counters.eager_steps == ids.shape[1]
    for mine, theirs in zip(captured.states, single.states):
        assert all(torch.equal(getattr(mine, name), getattr(theirs, name)) for name in ("fast", "slow", "mixed", "k", "v", "u"))
