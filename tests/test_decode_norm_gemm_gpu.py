"""The decode step of one sequence, whose projections form the residual sum and the norm that they read, against the step that
launches those by themselves: the same logits and state, bit for bit."""
import pytest
import torch

from warpstate_ai_b200 import WarpStateConfig, WarpStateLM
from warpstate_ai_b200.ops.gemm import check_device_errors
from warpstate_ai_b200.serve.engine import DecodeEngine


# narrowest and widest rows taken; widths whose columns leave worker threads idle; 14 partials, which are two rounds of loads (1280 x
# 4480); weights in tiles; a vocabulary that ends inside a slab
@pytest.mark.gpu
@pytest.mark.parametrize("d,ffn,packed,graph", [(64, 128, False, True), (640, 704, False, False), (1280, 4480, True, True),
                                                (1280, 4480, False, False), (1984, 1024, False, True), (2048, 7168, False, True),
                                                (2048, 1024, True, False)])
def test_norms_inside_the_projections_change_no_bit(d, ffn, packed, graph):
    batch = 1
    vocab, steps = 1000, 12
    cfg = WarpStateConfig(vocab_size=vocab, d_model=d, n_heads=d // 64, n_cores=2, logical_depth=3, ffn_hidden=ffn,
                          chunk_size=128, gradient_checkpointing=False, parallel_memory=True)
    torch.manual_seed(d)
    with torch.device("cuda"):
        model = WarpStateLM(cfg)
    with torch.no_grad():
        model.depth_scale.normal_(0, 0.1)
        model.depth_bias.normal_(0, 0.1)
    model.eval().requires_grad_(False)
    ids = torch.randint(0, vocab, (batch, 120 + steps), device="cuda")
    inside = DecodeEngine(model, pack_weights=packed, use_cuda_graph=graph)
    apart = DecodeEngine(model, pack_weights=packed, use_cuda_graph=graph)
    for engine in (inside, apart):
        engine.new_state(batch)
        assert engine._norm_in_gemm
    apart._norm_in_gemm = False
    for engine in (inside, apart):
        engine.prefill(ids[:, :120])
    for t in range(120, 120 + steps):                       # over the end of a chunk
        assert torch.equal(inside.step(ids[:, t]), apart.step(ids[:, t])), t
    check_device_errors()
    for mine, theirs in zip(inside.states, apart.states):
        assert all(torch.equal(getattr(mine, name), getattr(theirs, name)) for name in ("k", "v", "u", "fast", "slow", "mixed"))
    if graph:      # and two sequences are launched one by one
        assert inside.graph_counters.kernels_per_replay == 5 * 3 + 1 and apart.graph_counters.kernels_per_replay == 7 * 3 + 2
    inside.new_state(2)
    assert not inside._norm_in_gemm
