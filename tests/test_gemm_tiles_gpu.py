"""BF16 results and kept logits leave the CTA-pair kernel through shared memory: edges of tiles in rows and columns, row
factors, and views of a wider buffer whose other columns stay as they are."""
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(256, 8, 1024), (257, 264, 1024), (300, 1000, 2048), (511, 40, 1088), (640, 296, 64)])
def test_bf16_results(m, n, k):
    from warpstate_ai_b200.ops import _ext, gemm
    _ext.require()
    torch.manual_seed(m)
    x = torch.randn(m, k, device="cuda").bfloat16()
    w = (torch.randn(n, k, device="cuda") / k ** 0.5).bfloat16()
    factor = torch.rand(m, device="cuda") + 0.5
    flag = gemm.error_flag(torch.device("cuda"))
    for rows, operand, mn in ((factor, w, False), (None, w.t().contiguous(), True)):
        wide = torch.randn(m, n + 16, device="cuda").bfloat16()
        before = wide.clone()
        torch.ops.ws_b200.gemm(x, operand, False, mn, 0, m, n, k, wide[:, :n], None, None, rows, 1.0, 0.0, flag)
        gemm.check_device_errors()
        want = x.double() @ w.double().T * (1.0 if rows is None else rows.double()[:, None])
        # one rounding to BF16 of an FP32 sum of k exact products
        bound = 2.0 ** -8 * want.abs() + k * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)
        assert ((wide[:, :n].double() - want).abs() <= bound).all(), mn
        assert torch.equal(wide[:, n:], before[:, n:])


@pytest.mark.gpu
@pytest.mark.parametrize("rows,vocab,keep", [(256, 1000, 256), (300, 520, 256), (300, 520, 300), (513, 264, 512)])
def test_kept_logits_and_label_log_probabilities(rows, vocab, keep):
    from warpstate_ai_b200.ops import _ext, gemm
    _ext.require()
    torch.manual_seed(rows)
    d = 256
    hidden = torch.randn(rows, d, device="cuda").bfloat16()
    weight = (torch.randn(vocab, d, device="cuda") * 0.2).bfloat16()
    labels = torch.randint(0, vocab, (rows,), device="cuda")
    labels[:6] = torch.tensor([0, 31, 32, vocab - 1, vocab - 2, 255], device="cuda")
    logp, lse, _, count, _, _, logits = torch.ops.ws_b200.lm_head_fwd_labelled(hidden, weight, labels, -100, keep,
                                                                               gemm.error_flag(torch.device("cuda")))
    gemm.check_device_errors()
    exact = hidden.double() @ weight.double().T
    assert int(count) == rows and logits.shape == (keep, vocab)
    bound = 2.0 ** -8 * exact.abs() + d * 2.0 ** -24 * (hidden.double().abs() @ weight.double().abs().T)
    assert ((logits.double() - exact[:keep]).abs() <= bound[:keep]).all()
    # the head works on logits rounded to BF16; a sum of `vocab` exponentials and a logarithm in FP32 behind that
    rounded = (hidden.float() @ weight.float().T).bfloat16().double()
    want = torch.log_softmax(rounded, dim=-1).gather(1, labels[:, None])[:, 0]
    assert torch.allclose(logp.double(), want, rtol=0, atol=float(2.0 ** -8 * exact.abs().max()))
    assert torch.allclose(lse.double(), torch.logsumexp(rounded, dim=-1), rtol=0, atol=1e-3)


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(256, 264, 64), (300, 1000, 512), (2000, 1096, 1024)])
def test_tiles_carry_what_rows_would(m, n, k):
    """Bit for bit the results of the single-CTA kernel, which stores row by row; kept logits are the head's product."""
    from warpstate_ai_b200.ops import _ext, gemm
    lib = _ext.cdll()
    torch.manual_seed(n)
    x, w = torch.randn(m, k, device="cuda").bfloat16(), torch.randn(n, k, device="cuda").bfloat16()
    try:
        lib.ws_gemm_set_pair_mode(1)
        pair = gemm.linear(x, w)
        kept = torch.ops.ws_b200.lm_head_fwd_labelled(x, w, torch.zeros(m, dtype=torch.long, device="cuda"), -100, m,
                                                      gemm.error_flag(x.device))[-1]
        lib.ws_gemm_set_pair_mode(0)
        assert torch.equal(pair, gemm.linear(x, w)) and torch.equal(kept, pair)
    finally:
        lib.ws_gemm_set_pair_mode(-1)
    gemm.check_device_errors()
