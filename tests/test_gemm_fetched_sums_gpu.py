"""Weight gradients of few tokens and many tiles: the old sums are fetched, added to and stored instead of reduced into, with the same bits."""
import pytest
import torch

from warpstate_ai_b200.ops import _ext, gemm


# at least four rounds of 256 x 256 tiles: the shortest contraction that takes it, a ragged one, ragged gradients in views of wider buffers, the
# longest; and sums beyond L2 behind a shorter contraction
@pytest.mark.gpu
@pytest.mark.parametrize("tokens,shapes", [(512, [(5120, 4096)]), (520, [(4872, 4200)]), (1000, [(2560, 2048), (5000, 1096), (1288, 5000), (264, 1280)]),
                                           (1536, [(5120, 4096)]), (256, [(8200, 4104)])])
@pytest.mark.parametrize("alpha", [1.0, 0.3])
def test_fetched_sums_equal_the_single_cta_kernels(tokens, shapes, alpha):
    _ext.require()
    torch.manual_seed(tokens)
    dys = [torch.randn(tokens, n, device="cuda").bfloat16() for n, _ in shapes]
    xs = [torch.randn(tokens, k, device="cuda").bfloat16() for _, k in shapes]
    before = [torch.randn(n, k + 8, device="cuda") for n, k in shapes]
    results = []
    try:
        for mode in (1, 0):
            _ext.cdll().ws_gemm_set_pair_mode(mode)
            sums = [b.clone() for b in before]
            views = [w[:, :k] for w, (_, k) in zip(sums, shapes)]
            if len(shapes) > 1 and alpha == 1.0:
                torch.ops.ws_b200.grad_weight_group(dys, xs, views, [1.0] * len(shapes), gemm.error_flag(torch.device("cuda")))
            else:
                for dy, x, view in zip(dys, xs, views):
                    gemm.grad_weight_accumulate(dy, x, view, accumulate=True, alpha=alpha)
            results.append(sums)
    finally:
        _ext.cdll().ws_gemm_set_pair_mode(-1)
    gemm.check_device_errors()
    for mine, theirs, old in zip(*results, before):
        assert torch.equal(mine, theirs) and not torch.equal(mine, old)


# the same gradient twice; two halves of the columns of one; rows that two share
@pytest.mark.gpu
@pytest.mark.parametrize("places", [lambda g: (g[:, :2048], g[:, :2048]), lambda g: (g[:, :2048], g[:, 2048:]), lambda g: (g[:8192, :2048], g[2048:, :2048])])
def test_gradients_of_a_group_that_share_memory(places):
    """Products and sums of small whole numbers, so that their order does not matter."""
    torch.manual_seed(2)
    tokens = 1024
    total = torch.randint(-50, 50, (10240, 4096), device="cuda").float()
    grads = places(total)
    dys = [torch.randint(-1, 2, (tokens, g.shape[0]), device="cuda").bfloat16() for g in grads]
    xs = [torch.randint(-1, 2, (tokens, g.shape[1]), device="cuda").bfloat16() for g in grads]
    want = total.clone()
    for g, dy, x in zip(places(want), dys, xs):
        g += dy.float().t() @ x.float()
    torch.ops.ws_b200.grad_weight_group(dys, xs, list(grads), [1.0] * len(grads), gemm.error_flag(total.device))
    gemm.check_device_errors()
    assert torch.equal(total, want)
