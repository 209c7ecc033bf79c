"""RMSNorm backward over row counts at the edges of its steps, blocks and rings, against 64 bits."""
import pytest
import torch

from warpstate_ai_b200.ops import _ext

U = 2.0 ** -24


def _reference(dz, x, rstd, w, dres, scale):
    g, h = dz.double(), x.double() * rstd.double()[:, None]
    terms = g * w.double() * h
    mean, size = terms.mean(1, keepdim=True), terms.abs().mean(1, keepdim=True)
    dx = rstd.double()[:, None] * (g * w.double() - h * mean)
    bound = rstd.double()[:, None] * ((g * w.double()).abs() + h.abs() * size)
    if dres is not None:
        dx, bound = dx + dres.double(), bound + dres.double().abs()
    if scale is not None:
        dx, bound = dx * (1 + scale.double()), bound * (1 + scale.double()).abs()
    return dx, bound, (g * h).sum(0), (g * h).abs().sum(0)


# one row, an odd one, the last count with two rows to a step and the first with one, a block's second and fifth step, full and partial warps
@pytest.mark.gpu
@pytest.mark.parametrize("rows,d", [(1, 128), (3, 2048), (592, 640), (593, 640), (889, 2048), (1780, 1280), (4000, 384)])
@pytest.mark.parametrize("dtype,shift", [(torch.float32, 0), (torch.bfloat16, 0), (torch.bfloat16, 4)])
def test_against_64_bits(rows, d, dtype, shift):
    _ext.require()
    torch.manual_seed(rows)

    def at(t):   # BF16 rows from any 8 bytes on
        return torch.empty(t.numel() + shift, device="cuda", dtype=t.dtype)[shift:].view_as(t).copy_(t) if t.dtype == torch.bfloat16 else t

    r = lambda *s: torch.randn(*s, device="cuda")  # noqa: E731
    dz, x, dres = at(r(rows, d).bfloat16()), at(r(rows, d).to(dtype)), at(r(rows, d).to(dtype))
    rstd, w, scale, bias = torch.rand(rows, device="cuda") + 0.5, r(d), r(d), r(d)
    # up to eight products and sums a thread, five shuffles, eight warps, and a dozen roundings around them
    error = 40 * U
    out = 2.0 ** -8 if dtype == torch.bfloat16 else 0.0
    for res, sc, low in ((dres, scale, False), (None, None, True)):
        dx, dxb, dw = torch.ops.ws_b200.rmsnorm_bwd(dz, x, rstd, w, res, sc, low)
        want, bound, dw_want, dw_bound = _reference(dz, x, rstd, w, res, sc)
        assert ((dx.double() - want).abs() <= error * bound + out * (want.abs() + error * bound)).all()
        if low:
            assert ((dxb.double() - want).abs() <= error * bound + 2.0 ** -8 * (want.abs() + error * bound)).all()
        assert ((dw.double() - dw_want).abs() <= (rows / 888 + 40) * U * dw_bound).all()
    if dtype == torch.float32:
        dx, grads = torch.ops.ws_b200.rmsnorm_bwd_mod(dz, None, rstd, w, dres, scale, bias, x)
        mod = x.double() * (1 + scale.double()) + bias.double()
        h_size = (x.double() * (1 + scale.double())).abs() + bias.double().abs()   # a sum that may cancel
        before, bound, dw_want, dw_bound = _reference(dz, mod, rstd, w, dres, None)
        _, wide, _, dw_wide = _reference(dz, h_size, rstd, w, dres, None)
        bound = torch.maximum(bound, wide)
        assert ((dx.double() - before * (1 + scale.double())).abs() <= error * bound * (1 + scale.double()).abs()).all()
        sums = (rows / 592 + 40) * U
        assert ((grads[0].double() - dw_want).abs() <= sums * torch.maximum(dw_bound, dw_wide)).all()
        got = {1: (before.sum(0), bound.sum(0)), 2: ((before * x.double()).sum(0), (bound * x.double().abs()).sum(0))}
        for k, (want, size) in got.items():
            assert ((grads[k].double() - want).abs() <= (sums + error) * size).all(), k
