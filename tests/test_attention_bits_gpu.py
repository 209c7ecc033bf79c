"""The backward pass of the attention and of the memories keeps its bits from version to version: an ulp here moves every gradient of the
blocks before it.  Digests of results on inputs that are computed from a counter, recorded with the one-block-per-unit form of the
scan and the one-CTA-per-tile form of the attention (CUDA 12.9)."""
import ctypes

import pytest
import torch

from warpstate_ai_b200.ops import _ext, attention, gemm

MASK = (1 << 32) - 1


def counted(salt, shape, scale, shift=0.0):
    """FP32 in [shift - scale, shift + scale), the same everywhere: exact integer and floating point operations on a counter."""
    count = 1
    for n in shape:
        count *= n
    x = torch.arange(count, device="cuda", dtype=torch.int64) + (salt << 20)
    for factor in (0x9E3779B1, 0x85EBCA77):
        x = (x * factor) & MASK
        x ^= x >> 15
    return ((x >> 8).float() * 2.0 ** -23 - 1.0).mul_(scale).add_(shift).view(shape)


def digest(t):
    bits = t.contiguous().view(torch.int16 if t.element_size() == 2 else torch.int32).flatten().long()
    weight = (torch.arange(bits.numel(), device=bits.device) * 0x9E3779B1 & MASK) | 1
    return int((bits * weight).sum()) & MASK


def scan(batch, chunks, heads):
    _ext.require()
    pointer = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    shape = (batch, chunks, heads, 4096)
    g, w = counted(1, shape, 1.0), counted(2, shape, 0.05)
    logits = [counted(3, (heads,), 1.0, 2.2), counted(4, (heads,), 1.0, 4.6), counted(5, (heads,), 1.0)]
    out, partials = torch.empty(shape, device="cuda", dtype=torch.bfloat16), torch.empty(batch * heads * 16, 3, device="cuda")
    assert _ext.cdll().ws_memory_scan_bwd(pointer(g), pointer(w), *map(pointer, logits), pointer(out), pointer(partials), batch, chunks, heads,
                                          ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    return digest(out), digest(partials)


# groups of 16 chunks: one, a ragged one, several with a ragged last one
@pytest.mark.gpu
@pytest.mark.parametrize("batch,chunks,heads,want", [(4, 16, 32, (240920067, 4255260269)), (2, 7, 20, (337001864, 1423111150)),
                                                     (1, 40, 8, (2012217170, 2247772373))])
def test_reverse_scan(batch, chunks, heads, want):
    assert scan(batch, chunks, heads) == want


def backward(batch, tokens, heads):
    ops, flag = torch.ops.ws_b200, gemm.error_flag(torch.device("cuda", torch.cuda.current_device()))
    rope = attention.rope_table(flag.device, pair_major=True)
    d = heads * 64
    qkvgu = counted(6, (batch * tokens, 5 * d), 1.6).bfloat16()
    dy = counted(7, (batch * tokens, d), 0.02).bfloat16()
    logits = [counted(8, (heads,), 1.0, 2.2), counted(9, (heads,), 1.0, 4.6), counted(10, (heads,), 1.0)]
    writes = ops.chunk_writes(qkvgu, rope, batch, tokens, heads, flag)
    states = ops.memory_scan(writes, *logits, True, False, None, None)[0]
    dqkvgu, partials = ops.attn_bwd(qkvgu, dy, states, writes, rope, *logits, batch, tokens, heads, flag)
    gemm.check_device_errors()
    return digest(dqkvgu), digest(partials)


# a tile for some of the CTAs, several tiles for each
@pytest.mark.gpu
@pytest.mark.parametrize("batch,tokens,heads,want", [(2, 512, 8, (1284358552, 4244229321)), (3, 1152, 20, (4009705236, 1860216500)),
                                                     (4, 2048, 32, (3996549729, 4087909000))])
def test_attention_backward(batch, tokens, heads, want):
    assert backward(batch, tokens, heads) == want
