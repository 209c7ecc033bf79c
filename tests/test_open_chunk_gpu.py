"""The chunk that a prompt ends in: the persistent attention kernel, whose low softmax terms go to their product through TMEM, gives the
bits of the one-tile-per-CTA kernel, which forms them in a second pass through shared memory."""
import pytest
import torch

from warpstate_ai_b200.ops import _ext, attention, gemm


# one position and 127 of them, edges of a warp's rows, prompts without and with complete chunks, and several tiles to a CTA
@pytest.mark.gpu
@pytest.mark.parametrize("batch,seq,heads", [(1, 1, 2), (1, 31, 3), (2, 33, 1), (1, 127, 2), (3, 129, 4), (1, 300, 32), (2, 255, 5), (5, 700, 16), (40, 200, 8)])
def test_open_chunk(batch, seq, heads):
    _ext.require()
    lib = _ext.cdll()
    torch.manual_seed(seq)
    qkvgu = (torch.randn(batch * seq, 5 * heads * 64, device="cuda") * 1.5).bfloat16()
    rope = attention.rope_table(qkvgu.device, pair_major=True)
    logits = [torch.randn(heads, device="cuda") for _ in range(3)]
    zeros = lambda *s, dtype=torch.bfloat16: torch.zeros(batch, heads, *s, device="cuda", dtype=dtype)  # noqa: E731
    results = []
    try:
        for mode in (0, 1, 1):
            lib.ws_attn_set_stream_mode(mode)
            state = [zeros(64, 64, dtype=torch.float32), zeros(64, 64, dtype=torch.float32), zeros(64, 64), *(zeros(128, 64) for _ in range(3))]
            results.append((torch.ops.ws_b200.attn_prefill(qkvgu, rope, *logits, batch, seq, heads, *state, gemm.error_flag(qkvgu.device)), *state))
    finally:
        lib.ws_attn_set_stream_mode(-1)
    gemm.check_device_errors()
    for other in results[1:]:
        assert all(torch.equal(a, b) for a, b in zip(results[0], other))
    assert float(results[0][0].abs().max()) > 0
