"""Weight gradients of the CTA-pair kernel: sums (beta 1) leave as bulk reductions, overwrites (0) as stores, anything else row
by row; grouped problems of ragged sizes, in views of a wider buffer whose other columns stay as they are."""
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("betas", [(1.0, 1.0, 1.0), (0.0, 1.0, 0.5), (0.0, 0.0, 2.0)])
@pytest.mark.parametrize("tokens", [8, 200, 1024])
def test_accumulated_stored_and_scaled_gradients(tokens, betas):
    from warpstate_ai_b200.ops import _ext, gemm
    _ext.require()
    torch.manual_seed(tokens)
    shapes = [(256, 64), (264, 328), (1000, 136)]          # (rows, columns) of the gradient: one tile, ragged ones
    dys = [torch.randn(tokens, n, device="cuda").bfloat16() for n, _ in shapes]
    xs = [torch.randn(tokens, k, device="cuda").bfloat16() for _, k in shapes]
    wide = [torch.randn(n, k + 8, device="cuda") for n, k in shapes]
    before = [w.clone() for w in wide]
    if betas[0] == 0.0:
        wide[0][:, :64] = float("nan")                      # an overwritten gradient is not read
    flag = gemm.error_flag(torch.device("cuda"))
    torch.ops.ws_b200.grad_weight_group(dys, xs, [w[:, :k] for w, (_, k) in zip(wide, shapes)], list(betas), flag)
    gemm.check_device_errors()
    for dy, x, w, old, beta, (_, k) in zip(dys, xs, wide, before, betas, shapes):
        product = dy.double().T @ x.double()
        want = product + (beta * old[:, :k].double() if beta else 0.0)
        # FP32 sums of `tokens` exact products: at most tokens * 2^-24 of the sum of their magnitudes, a tenth of it in the mean
        bound = tokens * 2.0 ** -24 * (dy.double().abs().T @ x.double().abs()) + 2.0 ** -22 * want.abs() + 1e-30
        assert ((w[:, :k].double() - want).abs() <= bound).all(), beta
        assert torch.equal(w[:, k:], old[:, k:])


@pytest.mark.gpu
@pytest.mark.parametrize("accumulate", [True, False])
def test_a_bulk_reduction_is_a_read_an_addition_and_a_write(accumulate):
    """Bit for bit the gradients of the single-CTA kernel, whose threads do that."""
    from warpstate_ai_b200.ops import _ext, gemm
    lib = _ext.cdll()
    torch.manual_seed(1)
    dy, x = torch.randn(1000, 520, device="cuda").bfloat16(), torch.randn(1000, 328, device="cuda").bfloat16()
    before = torch.randn(520, 328, device="cuda")
    results = []
    try:
        for mode in (1, 0):
            lib.ws_gemm_set_pair_mode(mode)
            grad = before.clone()
            gemm.grad_weight_accumulate_group([(dy, x, grad, accumulate)])
            gemm.grad_weight_accumulate(dy, x, grad, accumulate=True, alpha=0.3)
            results.append(grad)
    finally:
        lib.ws_gemm_set_pair_mode(-1)
    gemm.check_device_errors()
    assert torch.equal(*results)
