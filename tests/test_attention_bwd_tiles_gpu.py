"""The attention backward's CTAs go from tile to tile through buffers that trade places every time: what a tile gives does not depend
on which of its CTA's tiles it is."""
import pytest
import torch


# 32 tiles a sequence over 296 CTAs (two per SM): 24 CTAs with a second tile; the third, with which the buffers are in their third places;
# a fourth for all but a few, in the first places again
@pytest.mark.gpu
@pytest.mark.parametrize("sequences", [10, 20, 37])
def test_a_tile_gives_the_same_whichever_tile_of_its_cta_it_is(sequences):
    from test_attention_gpu import make_core
    from warpstate_ai_b200.ops import attention
    from warpstate_ai_b200.ops.gemm import check_device_errors
    torch.manual_seed(sequences)
    heads, length = 8, 512
    core = make_core(heads)
    qkvgu = (torch.randn(sequences, length, 5 * 64 * heads, device="cuda") * 1.5).bfloat16()
    dy = torch.randn(sequences, length, 64 * heads, device="cuda").bfloat16()

    def gradient(part):
        n = qkvgu[part].shape[0]
        packed, dout = qkvgu[part].reshape(n * length, -1), dy[part].reshape(n * length, -1)
        _, saved = attention.forward(packed, core, n, length)
        return attention.backward(dout, packed, saved, core, n, length)[0].view(n, length, -1)

    together = gradient(slice(None))
    check_device_errors()
    for first in range(0, sequences, 9):            # at most 288 tiles: one for each CTA
        part = slice(first, first + 9)
        assert torch.equal(together[part], gradient(part)), first
