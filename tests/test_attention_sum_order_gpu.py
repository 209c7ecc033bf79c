"""A row's softmax sum goes through its columns in order, whatever the number of threads that share the row."""
import pytest
import torch

from warpstate_ai_b200.ops import _ext, gemm


@pytest.mark.gpu
@pytest.mark.parametrize("stream_form", [0, 1])
@pytest.mark.parametrize("batch,tokens,prompt", [(3, 256, False), (2, 256, True), (2, 100, True)])
def test_small_terms_behind_large_ones_are_lost_one_by_one(stream_form, batch, tokens, prompt):
    """Columns 0 and 1 weigh 1 each, every other column exp(-17) < 2 ** -24: behind the two, a pair of them is less than half an ulp of
    the sum, which stays 2.  Added up on their own first they would not be lost, and 1 / sum would be below 1 / 2.  The two values
    are (1 + 2 ** -7) and (1 + 2 ** -6), the others 0, so that half their sum lies in the middle of two BF16 numbers and goes to the
    even one, 1 + 2 ** -6; with any smaller factor it goes to the other.  No rotation, an open gate: every step before is exact."""
    heads = 4
    d = heads * 64
    rows = torch.arange(batch * tokens, device="cuda") % tokens % 128
    qkvgu = torch.zeros(batch * tokens, 5, heads, 64, device="cuda")
    qkvgu[:, 0, :, 0] = 8.0
    qkvgu[:, 1, :, 0] = torch.where(rows < 2, 0.0, -17.0)[:, None]
    qkvgu[rows == 0, 2] = 1.0 + 2.0 ** -7
    qkvgu[rows == 1, 2] = 1.0 + 2.0 ** -6
    qkvgu[:, 3] = 100.0
    qkvgu = qkvgu.view(batch * tokens, 5 * d).bfloat16()
    rope = torch.zeros(64 // 2, 128, 2, device="cuda")
    rope[..., 0] = 1.0
    flag, ops = gemm.error_flag(qkvgu.device), torch.ops.ws_b200
    logits = [torch.zeros(heads, device="cuda")] * 3
    lib = _ext.cdll()
    try:
        lib.ws_attn_set_stream_mode(stream_form)
        if prompt:
            state = [torch.zeros(batch, heads, 64, 64, device="cuda") for _ in range(2)] + [torch.zeros(batch, heads, 64, 64, device="cuda").bfloat16()]
            state += [torch.zeros(batch, heads, 128, 64, device="cuda").bfloat16() for _ in range(3)]
            y = ops.attn_prefill(qkvgu, rope, *logits, batch, tokens, heads, *state, flag)
        else:
            states = torch.zeros(batch, tokens // 128, heads, 64, 64, device="cuda").bfloat16()
            y = ops.attn_fwd(qkvgu, states, rope, batch, tokens, heads, flag)
    finally:
        lib.ws_attn_set_stream_mode(-1)
    gemm.check_device_errors()
    want = torch.where(rows == 0, 1.0 + 2.0 ** -7, 1.0 + 2.0 ** -6)[:, None].expand(-1, d)
    assert torch.equal(y.float(), want)
