"""Residual + norm of a decode step: the sums, the modulation and the squares with their roundings as they are written out, bit for
bit, for rows that the short kernel holds (d <= 2048) and longer ones, with fewer partials than one round of loads and more."""
import pytest
import torch

THREADS = 256      # of the sum of squares: thread t adds columns 4 t .. 4 t + 3 of every block of 1024


def fma(a, b, c):
    """One rounding: the product of two FP32 values is exact in FP64, and so is the sum but for cases of 2^-29."""
    return (a.double() * b.double() + c.double()).float()


def reference(x, partials, scale, bias, w, eps):
    v = x.clone()
    for p in partials:
        v = v + p
    if scale is not None:
        v = fma(v, 1.0 + scale, bias)
    batch, d = v.shape
    a, b, c, e = torch.nn.functional.pad(v, (0, -d % (4 * THREADS))).view(batch, -1, THREADS, 4).unbind(-1)
    squares = fma(e, e, fma(c, c, fma(a, a, b * b)))
    sums = squares[:, 0]
    for block in squares[:, 1:].unbind(1):
        sums = sums + block
    sums = sums.view(batch, THREADS // 32, 32)
    lane = torch.arange(32, device=v.device)
    for o in (16, 8, 4, 2, 1):
        sums = sums + sums[..., lane ^ o]
    total = torch.zeros(batch, device=v.device)
    for warp in sums[..., 0].unbind(1):
        total = total + warp
    return v, (v * torch.rsqrt(total / d + eps)[:, None] * w).bfloat16()


@pytest.mark.gpu
@pytest.mark.parametrize("modulated", [False, True])
@pytest.mark.parametrize("d,splits", [(256, 1), (1024, 8), (2048, 4), (2048, 17), (4096, 3)])
def test_bit_for_bit(d, splits, modulated):
    """Powers of two, so that the mean needs no rounding.  An ulp of a sum of squares shows in few of the BF16 results: there
    are enough rows here for several."""
    from warpstate_ai_b200.ops import _ext
    _ext.require()
    torch.manual_seed(d + splits)
    batch = 64
    out = torch.empty(batch, d, device="cuda", dtype=torch.bfloat16)
    for _ in range(200 if d > 256 else 800):
        x = torch.randn(batch, d, device="cuda") * 0.3
        partials = torch.randn(splits, batch, d, device="cuda") * 0.1
        scale, bias, w = (torch.randn(d, device="cuda") * 0.05 for _ in range(3))
        mod = (scale, bias) if modulated else (None, None)
        want_x, want = reference(x, partials, *mod, w + 1, 1e-5)
        torch.ops.ws_b200.decode_reduce_norm(x, partials, None, None, *mod, w + 1, 1e-5, out)
        assert torch.equal(x, want_x) and torch.equal(out, want)


@pytest.mark.gpu
@pytest.mark.parametrize("d", [4, 256, 1280, 2044, 2048, 2052, 2176])
def test_widths_tokens_and_a_row_that_is_only_updated(d):
    from warpstate_ai_b200.ops import _ext
    _ext.require()
    torch.manual_seed(d)
    batch, vocab = 5, 9
    table, w = torch.randn(vocab, d, device="cuda"), torch.randn(d, device="cuda")
    scale, bias = torch.randn(2, d, device="cuda").mul_(0.1).unbind(0)
    token = torch.tensor([0, vocab - 1, 3, vocab + 5, -2], device="cuda")
    out = torch.empty(batch, d, device="cuda", dtype=torch.bfloat16)
    x = torch.empty(batch, d, device="cuda")
    torch.ops.ws_b200.decode_reduce_norm(x, None, token, table, scale, bias, w, 1e-5, out)
    want_x, want = reference(table[token.clamp(0, vocab - 1)], [], scale, bias, w, 1e-5)
    assert torch.equal(x, want_x)
    # one rounding to BF16, of a factor that is right to a few FP32 ulps
    assert ((out.double() - want.double()).abs() <= 2.0 ** -7 * want.double().abs()).all()
    partials = torch.randn(11, batch, d, device="cuda")
    torch.ops.ws_b200.decode_reduce_norm(x, partials, None, None, None, None, w, 1e-5, None)
    assert torch.equal(x, reference(want_x, partials, None, None, w, 1e-5)[0])
