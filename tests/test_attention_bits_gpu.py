"""The backward pass of the memories keeps its bits from version to version: an ulp here moves every gradient of the blocks before it.
Digests of results on inputs that are computed from a counter, recorded with the one-block-per-unit form of the scan (CUDA 12.9)."""
import ctypes

import pytest
import torch

from warpstate_ai_b200.ops import _ext

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
