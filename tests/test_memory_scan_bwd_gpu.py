"""The reverse scan of the memory states against the recurrences in 64 bits, and from writes that are not aligned to 16 bytes."""
import ctypes

import pytest
import torch

from warpstate_ai_b200.ops import _ext, gemm


def _pointer(t):
    return ctypes.c_void_p(t.data_ptr())


def _reference(g, w, df, ds, mix, sign=-1):
    """Gradients of the writes and the three sums per head; with absolute values and `sign` 1, what those are made of at most."""
    fast, slow = torch.zeros_like(w[:, 0]), torch.zeros_like(w[:, 0])
    seen = []
    for n in range(w.shape[1]):
        seen.append((fast, slow))
        fast, slow = df * fast + (1 - df) * w[:, n], ds * slow + (1 - ds) * w[:, n]
    a, b = torch.zeros_like(fast), torch.zeros_like(fast)
    grads, sums = torch.zeros_like(w), torch.zeros(3, w.shape[0], w.shape[2], dtype=w.dtype, device=w.device)
    for n in reversed(range(w.shape[1])):
        fast, slow = seen[n]
        grads[:, n] = (1 - df) * a + (1 - ds) * b
        sums += torch.stack([(a * (fast + sign * w[:, n])).sum(-1), (b * (slow + sign * w[:, n])).sum(-1), (g[:, n] * (fast + sign * slow)).sum(-1)])
        a, b = mix * g[:, n] + df * a, (1 - mix) * g[:, n] + ds * b
    return grads, sums


# one unit per CTA and several of them, groups of 16 chunks that are whole, ragged and more than one
@pytest.mark.gpu
@pytest.mark.parametrize("batch,chunks,heads", [(1, 1, 1), (2, 7, 3), (1, 16, 29), (2, 4, 32), (1, 17, 3), (1, 33, 2), (2, 24, 16)])
def test_against_64_bits(batch, chunks, heads):
    _ext.require()
    torch.manual_seed(chunks)
    shape = (batch, chunks, heads, 4096)
    g, w = torch.randn(shape, device="cuda"), torch.randn(shape, device="cuda")
    logits = torch.randn(3, heads, device="cuda")
    out = torch.empty(shape, device="cuda", dtype=torch.bfloat16)
    partials = torch.empty(batch * heads, 16, 3, device="cuda")
    assert _ext.cdll().ws_memory_scan_bwd(_pointer(g), _pointer(w), _pointer(logits[0]), _pointer(logits[1]), _pointer(logits[2]), _pointer(out),
                                          _pointer(partials), batch, chunks, heads, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    df, ds, mix = torch.sigmoid(logits.double())[:, None, :, None]
    grads, sums = _reference(g.double(), w.double(), df, ds, mix)
    most, terms = _reference(g.double().abs(), w.double().abs(), df, ds, mix, 1)
    # a chunk adds four roundings to a state or its gradient, the decays have a few of their own; the result is rounded to BF16
    error = (4 * chunks + 16) * 2.0 ** -24
    assert ((out.double() - grads).abs() <= 2.0 ** -8 * grads.abs() + error * most).all()
    # of the terms of a sum a thread adds 2 x chunks, and the block its 128 threads' in ten more roundings
    got = partials.double().view(batch, heads, 16, 3).sum(2).permute(2, 0, 1)
    assert ((got - sums).abs() <= (2 * error + (chunks + 10) * 2.0 ** -24) * terms).all()


@pytest.mark.gpu
def test_writes_at_any_float():
    _ext.require()
    torch.manual_seed(1)
    b, t, h = 2, 384, 4
    r = lambda *s: torch.randn(*s, device="cuda").bfloat16()  # noqa: E731
    from warpstate_ai_b200.ops.attention import rope_table
    qkvgu, dy, states = r(b * t, 5 * h * 64), r(b * t, h * 64), r(b, t // 128, h, 64, 64)
    writes = torch.randn(b * (t // 128) * h * 4096 + 2, device="cuda")
    logits = torch.randn(3, h, device="cuda")
    flag = gemm.error_flag(torch.device("cuda"))
    results = []
    for at in (0, 2):
        w = writes[at:at + writes.numel() - 2]
        w.copy_(torch.linspace(-1, 1, w.numel(), device="cuda"))
        results.append(torch.ops.ws_b200.attn_bwd(qkvgu, dy, states, w.view(b, t // 128, h, 64, 64), rope_table(qkvgu.device, pair_major=True),
                                                  *logits.unbind(0), b, t, h, flag))
    gemm.check_device_errors()
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])
