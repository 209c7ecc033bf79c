"""Products that fit the chip in one round of 256 x 128 tiles: the bits of the single-CTA kernel, over every epilogue that takes such tiles."""
import pytest
import torch

from warpstate_ai_b200.ops import _ext, gemm


def _both(run):
    results = []
    try:
        for mode in (1, 0):
            _ext.cdll().ws_gemm_set_pair_mode(mode)
            results.append(run())
    finally:
        _ext.cdll().ws_gemm_set_pair_mode(-1)
    gemm.check_device_errors()
    return results


# one tile, ragged rows and columns, a last half tile of 8 columns, the most tiles that are one round on 148 SMs and one more
@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(256, 8, 64), (300, 136, 256), (511, 264, 200), (1792, 1280, 1280), (256, 74 * 128, 128), (256, 74 * 128 + 8, 128)])
def test_products(m, n, k):
    _ext.require()
    torch.manual_seed(n)
    r = lambda *s: torch.randn(*s, device="cuda").bfloat16()  # noqa: E731
    x, w, resid, factor = r(m, k), r(n, k), torch.randn(m, n, device="cuda"), torch.rand(m, device="cuda")
    wt = w.t().contiguous()
    for run in (lambda: gemm.linear(x, w), lambda: gemm.linear(x, w, row_scale=factor), lambda: gemm.linear_f32(x, w),
                lambda: gemm.linear_residual(x, w, resid), lambda: gemm.grad_input(x, wt)):
        pair, single = _both(run)
        assert torch.equal(pair, single)


@pytest.mark.gpu
@pytest.mark.parametrize("m,h,k", [(256, 8, 64), (300, 200, 256), (256, 74 * 64, 128), (256, 74 * 64 + 8, 128), (1024, 688, 256)])
def test_swiglu(m, h, k):
    _ext.require()
    torch.manual_seed(h)
    r = lambda *s: torch.randn(*s, device="cuda").bfloat16()  # noqa: E731
    x, w, dy, down, packed = r(m, k), r(2 * h, k), r(m, k), r(k, h), r(m, 2 * h)
    pair, single = _both(lambda: gemm.linear_swiglu(x, w))
    assert all(torch.equal(a, b) for a, b in zip(pair, single))
    pair, single = _both(lambda: gemm.grad_input_swiglu(dy, down, packed))
    # the single-CTA kernel contracts the derivative's products in an order of its own
    assert torch.allclose(pair.float(), single.float(), rtol=2.0 ** -7, atol=2.0 ** -14)


@pytest.mark.gpu
@pytest.mark.parametrize("tokens,shapes", [(256, [(8, 8)]), (520, [(200, 136), (264, 256), (512, 72), (8, 600)]), (1024, [(1280, 256), (256, 256), (1376, 256), (256, 688)])])
@pytest.mark.parametrize("alpha,beta", [(1.0, 1), (0.5, 0)])
def test_weight_gradients(tokens, shapes, alpha, beta):
    _ext.require()
    torch.manual_seed(tokens)
    dys = [torch.randn(tokens, n, device="cuda").bfloat16() for n, _ in shapes]
    xs = [torch.randn(tokens, k, device="cuda").bfloat16() for _, k in shapes]
    before = [torch.randn(n, k, device="cuda") for n, k in shapes]

    def run():
        sums = [b.clone() for b in before]
        if beta and alpha == 1.0:
            torch.ops.ws_b200.grad_weight_group(dys, xs, sums, [1.0] * len(shapes), gemm.error_flag(torch.device("cuda")))
        else:
            for dy, x, g in zip(dys, xs, sums):
                gemm.grad_weight_accumulate(dy, x, g, accumulate=bool(beta), alpha=alpha)
        return sums

    pair, single = _both(run)
    assert all(torch.equal(a, b) for a, b in zip(pair, single))


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(128, 2048, 7168), (96, 1280, 4480)])
def test_pieces(m, n, k):
    """A product cut along k, whose pieces are half tiles, against 64 bits: one rounding of `pieces` FP32 sums of exact products."""
    _ext.require()
    torch.manual_seed(m)
    x, w, resid = torch.randn(m, k, device="cuda").bfloat16(), torch.randn(n, k, device="cuda").bfloat16(), torch.randn(m, n, device="cuda")
    got = gemm.linear_residual(x, w, resid)
    gemm.check_device_errors()
    want = resid.double() + x.double() @ w.double().T
    bound = (k + 8) * 2.0 ** -24 * (resid.double().abs() + x.double().abs() @ w.double().abs().T)
    assert ((got.double() - want).abs() <= bound).all()
