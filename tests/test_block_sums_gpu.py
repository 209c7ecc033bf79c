"""The small sums behind a block's backward pass, in one launch: the bits of the launches that add each of them up alone."""
import ctypes

import pytest
import torch

from warpstate_ai_b200.ops import _ext


# one head and 32 of them, one partial row, counts around the rounds of 128 parts, with and without a modulation's sums
@pytest.mark.gpu
@pytest.mark.parametrize("heads,batch,second,first,sums", [(1, 1, 1, 1, 1), (4, 2, 256, 129, 3), (20, 2, 444, 296, 3), (32, 8, 444, 444, 1), (3, 5, 33, 31, 3)])
def test_block_sums(heads, batch, second, first, sums):
    _ext.require()
    lib, d = _ext.cdll(), 64 * heads
    torch.manual_seed(second)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    a, b, scan = torch.randn(second, d, device="cuda"), torch.randn(sums, first, d, device="cuda"), torch.randn(batch * heads * 16, 3, device="cuda")
    logits = torch.randn(3, heads, device="cuda")
    one, many, grads = torch.empty(d, device="cuda"), torch.empty(sums, d, device="cuda"), torch.empty(3, heads, device="cuda")
    assert lib.ws_block_sums(p(a), second, p(one), p(b), first, sums, p(many), p(scan), p(logits[0]), p(logits[1]), p(logits[2]), batch, heads, p(grads), d,
                             stream) == 0
    for partial, got in ((a, one), *zip(b, many)):
        alone = torch.empty(d, device="cuda")
        assert lib.ws_colsum_finalize(p(partial), partial.shape[0], d, None, ctypes.c_float(0.0), p(alone), stream) == 0
        assert torch.equal(got, alone)
    assert torch.equal(grads, torch.ops.ws_b200.memory_logit_grads(scan, *logits.unbind(0), batch))
